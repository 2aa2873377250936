// The learned smoother's network: parameters, tensor-core inference, and the
// trainer (hand-written backward + Adam).  C ABI in include/mgsb.h
// (mgsb_mlp_*); no counterpart in the reference.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/mgsb.h"
#include "kernels_mlp.cuh"
#include "mlp.hpp"

using namespace mgsb;

struct mgsb_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    float *prm = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *loss = nullptr;
    uint8_t* img = nullptr;
    int adam_t = 0;
    // growable scratch: the rows of a training launch (at most kTrainChunk samples) and its samples' errors
    float *act = nullptr, *lsum = nullptr;
    int act_cap = 0;   // blocks of 128 samples
    float *X = nullptr, *T = nullptr, *Y = nullptr;
    size_t data_cap = 0;
    int32_t* werr = nullptr;
    ~mgsb_mlp();
};

mgsb_mlp::~mgsb_mlp() {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    for (void* p : {(void*)prm, (void*)m, (void*)v, (void*)grad, (void*)loss, (void*)img, (void*)act,
                    (void*)lsum, (void*)X, (void*)T, (void*)Y, (void*)werr})
        if (p) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
}

namespace {

mgsb_status mlp_err(mgsb_mlp* h, mgsb_status s, const char* fmt, ...) {
    if (h) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        h->err = buf;
    }
    return s;
}

#define MLP_CUDA(h, call)                                                                              \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess) return mlp_err(h, MGSB_CUDA_ERROR, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)
#define MLP_TRY(expr)                      \
    do {                                   \
        mgsb_status s_ = (expr);           \
        if (s_ != MGSB_OK) return s_;      \
    } while (0)

size_t mlp_tc_smem() { return mlp_tc_smem_bytes(); }

mgsb_status ensure_data(mgsb_mlp* h, size_t n) {
    if (n <= h->data_cap) return MGSB_OK;
    for (float** p : {&h->X, &h->T, &h->Y}) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    h->data_cap = 0;
    MLP_CUDA(h, cudaMalloc(&h->X, n * kMlpIn * sizeof(float)));
    MLP_CUDA(h, cudaMalloc(&h->T, n * kMlpOut * sizeof(float)));
    MLP_CUDA(h, cudaMalloc(&h->Y, n * kMlpOut * sizeof(float)));
    h->data_cap = n;
    return MGSB_OK;
}

mgsb_status ensure_act(mgsb_mlp* h, int samples) {
    const int nblk = train_blocks(std::min(samples, kTrainChunk));
    if (nblk <= h->act_cap) return MGSB_OK;
    if (h->act) cudaFree(h->act);
    if (h->lsum) cudaFree(h->lsum);
    h->act = h->lsum = nullptr;
    h->act_cap = 0;
    MLP_CUDA(h, cudaMalloc(&h->act, (size_t)kActRows * nblk * kGradLd * sizeof(float)));
    MLP_CUDA(h, cudaMalloc(&h->lsum, (size_t)nblk * kGradBlock * sizeof(float)));
    h->act_cap = nblk;
    return MGSB_OK;
}

mgsb_status repack(mgsb_mlp* h) {
    k_mlp_pack<<<(kMlpHid * kMlpHid + 255) / 256, 256, 0, h->stream>>>(h->prm, h->img);
    MLP_CUDA(h, cudaGetLastError());
    return MGSB_OK;
}

// Kernel launch that may start while the one before it finishes (both wait for it before they touch its results).
template <typename... KArgs, typename... Args>
cudaError_t launch_after(mgsb_mlp* h, void (*kernel)(KArgs...), int grid, int block, size_t smem, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Mean squared error over `nb` samples (rows 0..nb-1 of X/T, or sampled), kTrainChunk of them per launch pair.  With
// adam the parameters take the step and loss_out (optional) gets the loss; else the gradient is left in h->grad and
// the loss in h->loss.
mgsb_status launch_grad(mgsb_mlp* h, int nb, SampleOf sample, const AdamStep* step, float* loss_out) {
    MLP_TRY(ensure_act(h, nb));
    const float inv = 1.f / (float)(nb * kMlpOut);
    for (int at = 0; at < nb; at += kTrainChunk) {
        const int n = std::min(kTrainChunk, nb - at), nblk = train_blocks(n), ld = nblk * kGradLd;
        sample.first = at;
        MLP_CUDA(h, launch_after(h, k_mlp_fwd_bwd, nblk * (kGradBlock / kTrainSamples), kTrainThreads, sizeof(TrainSmem), n,
                                 sample, (const float*)h->X, (const float*)h->T, (const float*)h->prm, h->act, ld, h->lsum, inv));
        MLP_CUDA(h, launch_after(h, k_mlp_grad, kGradTiles, kGradThreads, sizeof(GradSmem), nblk, (const float*)h->act, ld,
                                 (const float*)h->lsum, at > 0 ? 1 : 0, at + n == nb ? 1 : 0, inv, h->grad, h->loss, loss_out,
                                 step ? h->prm : (float*)nullptr, h->m, h->v, step ? *step : AdamStep{}, h->werr));
    }
    return MGSB_OK;
}

// The training kernels' bounded waits.
mgsb_status check_waits(mgsb_mlp* h) {
    int32_t werr = 0;
    MLP_CUDA(h, cudaMemcpyAsync(&werr, h->werr, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    MLP_CUDA(h, cudaStreamSynchronize(h->stream));
    return werr ? mlp_err(h, MGSB_TIMEOUT, "network training: a bounded wait ran out") : MGSB_OK;
}

// Deterministic initialisation (uniform +-sqrt(6/(fan_in+fan_out)), zero biases).
void init_params(uint64_t seed, std::vector<float>& p) {
    p.assign(kMlpParams, 0.f);
    uint64_t z = seed;
    auto next = [&z]() {
        z += 0x9E3779B97F4A7C15ull;
        uint64_t x = z;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        x ^= x >> 31;
        return (double)(x >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int fan_out, int fan_in) {
        const double a = std::sqrt(6.0 / (fan_in + fan_out));
        for (int i = 0; i < fan_out * fan_in; ++i) p[off + i] = (float)((2.0 * next() - 1.0) * a);
    };
    fill(kOffW1, kMlpHid, kMlpIn);
    fill(kOffW2, kMlpHid, kMlpHid);
    fill(kOffW3, kMlpOut, kMlpHid);
}

}  // namespace

namespace mgsb {
const uint8_t* mlp_device_image(const mgsb_mlp* h) { return h ? h->img : nullptr; }
int mlp_device(const mgsb_mlp* h) { return h ? h->device : -1; }
}  // namespace mgsb

extern "C" {

int32_t mgsb_mlp_num_params(void) { return kMlpParams; }

mgsb_status mgsb_mlp_create(int32_t device, uint64_t seed, mgsb_mlp** out) {
    if (!out) return MGSB_INVALID_ARG;
    *out = nullptr;
    mgsb_mlp* h = new mgsb_mlp;
    h->device = device;
    auto fail = [&](mgsb_status s) {
        delete h;
        return s;
    };
    if (cudaSetDevice(device) != cudaSuccess) return fail(MGSB_CUDA_ERROR);
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(MGSB_CUDA_ERROR);
    const size_t pb = kMlpParams * sizeof(float);
    if (cudaMalloc(&h->prm, pb) || cudaMalloc(&h->m, pb) || cudaMalloc(&h->v, pb) || cudaMalloc(&h->grad, pb) ||
        cudaMalloc(&h->loss, sizeof(float)) || cudaMalloc(&h->img, kImgBytes) || cudaMalloc(&h->werr, sizeof(int32_t)))
        return fail(MGSB_OUT_OF_MEMORY);
    if (cudaFuncSetAttribute(k_mlp_fwd_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem)) ||
        cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem)) ||
        cudaFuncSetAttribute(k_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_tc_smem()))
        return fail(MGSB_CUDA_ERROR);
    std::vector<float> p;
    init_params(seed, p);
    if (cudaMemcpy(h->prm, p.data(), pb, cudaMemcpyHostToDevice) || cudaMemset(h->m, 0, pb) || cudaMemset(h->v, 0, pb) ||
        cudaMemset(h->werr, 0, sizeof(int32_t)))
        return fail(MGSB_CUDA_ERROR);
    if (repack(h) != MGSB_OK || cudaStreamSynchronize(h->stream) != cudaSuccess) return fail(MGSB_CUDA_ERROR);
    *out = h;
    return MGSB_OK;
}

mgsb_status mgsb_mlp_destroy(mgsb_mlp* h) {
    delete h;
    return MGSB_OK;
}

const char* mgsb_mlp_last_error(const mgsb_mlp* h) { return h ? h->err.c_str() : "null handle"; }

mgsb_status mgsb_mlp_set_params(mgsb_mlp* h, const float* params, int32_t n) {
    if (!h || !params || n != kMlpParams) return mlp_err(h, MGSB_INVALID_ARG, "expected %d parameters", kMlpParams);
    MLP_CUDA(h, cudaSetDevice(h->device));
    MLP_CUDA(h, cudaMemcpyAsync(h->prm, params, kMlpParams * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MLP_CUDA(h, cudaMemsetAsync(h->m, 0, kMlpParams * sizeof(float), h->stream));
    MLP_CUDA(h, cudaMemsetAsync(h->v, 0, kMlpParams * sizeof(float), h->stream));
    h->adam_t = 0;
    MLP_TRY(repack(h));
    MLP_CUDA(h, cudaStreamSynchronize(h->stream));
    return MGSB_OK;
}

mgsb_status mgsb_mlp_get_params(mgsb_mlp* h, float* params, int32_t n) {
    if (!h || !params || n != kMlpParams) return mlp_err(h, MGSB_INVALID_ARG, "expected %d parameters", kMlpParams);
    MLP_CUDA(h, cudaSetDevice(h->device));
    MLP_CUDA(h, cudaMemcpyAsync(params, h->prm, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    MLP_CUDA(h, cudaStreamSynchronize(h->stream));
    return MGSB_OK;
}

mgsb_status mgsb_mlp_forward(mgsb_mlp* h, const float* x, int32_t n, float* y) {
    if (!h || !x || !y || n < 0) return MGSB_INVALID_ARG;
    if (n == 0) return MGSB_OK;
    MLP_CUDA(h, cudaSetDevice(h->device));
    MLP_TRY(ensure_data(h, n));
    const int ntiles = (n + kMlpTile - 1) / kMlpTile;
    MLP_CUDA(h, cudaMemcpyAsync(h->X, x, (size_t)n * kMlpIn * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MLP_CUDA(h, cudaMemsetAsync(h->werr, 0, sizeof(int32_t), h->stream));
    int dev_sms = 148;
    cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, h->device);
    const int grid = std::min(ntiles, 2 * dev_sms);
    k_mlp_tc<<<grid, kMlpThreads, mlp_tc_smem(), h->stream>>>(n, ntiles, h->X, h->img, h->Y, h->werr);
    MLP_CUDA(h, cudaGetLastError());
    int32_t werr = 0;
    MLP_CUDA(h, cudaMemcpyAsync(&werr, h->werr, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    MLP_CUDA(h, cudaStreamSynchronize(h->stream));
    if (werr) return mlp_err(h, MGSB_TIMEOUT, "tensor-core MLP: a bounded wait ran out");
    // straight into the caller's array, which the driver stages: as fast as two pinned halves of this handle's own (0.34
    // and 0.35 ms a call on 100,000 rows), which cost a handle's first call 1 to 3 ms
    MLP_CUDA(h, cudaMemcpyAsync(y, h->Y, (size_t)n * kMlpOut * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    MLP_CUDA(h, cudaStreamSynchronize(h->stream));
    return MGSB_OK;
}

mgsb_status mgsb_mlp_loss_grad(mgsb_mlp* h, const float* x, const float* t, int32_t n, float* grad, float* loss) {
    if (!h || !x || !t || n <= 0) return MGSB_INVALID_ARG;
    MLP_CUDA(h, cudaSetDevice(h->device));
    MLP_TRY(ensure_data(h, n));
    MLP_CUDA(h, cudaMemcpyAsync(h->X, x, (size_t)n * kMlpIn * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MLP_CUDA(h, cudaMemcpyAsync(h->T, t, (size_t)n * kMlpOut * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MLP_CUDA(h, cudaMemsetAsync(h->werr, 0, sizeof(int32_t), h->stream));
    MLP_TRY(launch_grad(h, n, SampleOf{0, 0, n, 0, 0}, nullptr, nullptr));
    if (grad)
        MLP_CUDA(h, cudaMemcpyAsync(grad, h->grad, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    if (loss) MLP_CUDA(h, cudaMemcpyAsync(loss, h->loss, sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    return check_waits(h);
}

mgsb_status mgsb_mlp_train(mgsb_mlp* h, const float* x, const float* t, int64_t n, int32_t steps, int32_t batch,
                           float lr, uint64_t seed, float* losses) {
    if (!h || !x || !t || n <= 0 || steps <= 0 || batch <= 0 || n > INT32_MAX) return MGSB_INVALID_ARG;
    MLP_CUDA(h, cudaSetDevice(h->device));
    MLP_TRY(ensure_data(h, (size_t)n));
    MLP_CUDA(h, cudaMemcpyAsync(h->X, x, (size_t)n * kMlpIn * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MLP_CUDA(h, cudaMemcpyAsync(h->T, t, (size_t)n * kMlpOut * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MLP_TRY(ensure_act(h, batch));
    MLP_CUDA(h, cudaMemsetAsync(h->werr, 0, sizeof(int32_t), h->stream));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float* hist = nullptr;   // loss of every step, read back once at the end
    if (losses) MLP_CUDA(h, cudaMalloc(&hist, (size_t)steps * sizeof(float)));
    struct Free {
        float* p;
        ~Free() { if (p) cudaFree(p); }
    } free_hist{hist};
    for (int s = 0; s < steps; ++s) {
        // cosine decay of the step size to 10 %
        const float lr_s = lr * (0.55f + 0.45f * std::cos(3.14159265f * (float)s / (float)steps));
        ++h->adam_t;
        const float bc1 = 1.f - std::pow(b1, (float)h->adam_t), bc2 = 1.f - std::pow(b2, (float)h->adam_t);
        const AdamStep step{lr_s, b1, b2, eps, bc1, bc2};
        MLP_TRY(launch_grad(h, batch, SampleOf{1, 0, (int)n, seed, (uint64_t)s}, &step, losses ? hist + s : nullptr));
    }
    MLP_CUDA(h, cudaGetLastError());
    MLP_TRY(repack(h));
    if (losses)
        MLP_CUDA(h, cudaMemcpyAsync(losses, hist, (size_t)steps * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    return check_waits(h);
}

}  // extern "C"
