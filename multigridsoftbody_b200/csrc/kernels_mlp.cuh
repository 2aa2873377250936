// Per-vertex MLP of the learned smoother: 9 features -> 64 -> 64 -> 3, GELU,
// BF16 weights and activations as tensor-core operands, FP32 accumulation.
//
//   inference  k_mlp_tc: tcgen05.mma (kind::f16, BF16 x BF16 -> FP32 in TMEM),
//              the weights staged in shared memory by a bulk async copy (TMA
//              engine), the rows' features rounded into the operand tile, one CTA
//              per 128-row tile, the three layers chained through TMEM ->
//              registers (bias, GELU) -> shared memory.
//   training   k_mlp_fwd_bwd: SIMT forward + hand-written backward with the same
//              BF16 rounding of the weights and activations, FP32 math;
//              k_mlp_grad: the weight gradients from its rows, summed in a fixed
//              order, and the Adam step.
//
// Parameter vector (FP32 master copy, 4,995 floats):
//   W1[64][9]  b1[64]  W2[64][64]  b2[64]  W3[3][64]  b3[3]
// Device image for the tensor cores (bf16, K-major, no swizzle, "interleaved"
// core matrices of 8 rows x 16 bytes):
//   W1 64x16 (K padded 9->16 with zeros) | W2 64x64 | W3 16x64 (rows padded
//   3->16 with zeros) | b1[64] b2[64] b3[16] (fp32)
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace mgsb {
namespace {

constexpr int kMlpIn = 9, kMlpInPad = 16, kMlpHid = 64, kMlpOut = 3, kMlpOutPad = 16;
constexpr int kMlpTile = 128;   // rows per tensor-core tile (MMA M)
constexpr int kMlpParams = kMlpHid * kMlpIn + kMlpHid + kMlpHid * kMlpHid + kMlpHid + kMlpOut * kMlpHid + kMlpOut;
// parameter offsets
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kMlpHid * kMlpIn, kOffW2 = kOffB1 + kMlpHid,
              kOffB2 = kOffW2 + kMlpHid * kMlpHid, kOffW3 = kOffB2 + kMlpHid, kOffB3 = kOffW3 + kMlpOut * kMlpHid;
static_assert(kOffB3 + kMlpOut == kMlpParams, "parameter layout");
// image offsets (bytes)
constexpr int kImgW1 = 0, kImgW2 = kImgW1 + kMlpHid * kMlpInPad * 2, kImgW3 = kImgW2 + kMlpHid * kMlpHid * 2,
              kImgB = kImgW3 + kMlpOutPad * kMlpHid * 2, kImgBytes = kImgB + (2 * kMlpHid + kMlpOutPad) * 4;
constexpr int kTileBytes = kMlpTile * kMlpInPad * 2;   // one feature tile: 4 KiB

// Byte offset of element (row, k) in a K-major interleaved tile of K columns:
// 8-row groups of (K/8) core matrices, each core matrix 8 rows x 16 bytes.
__host__ __device__ constexpr int interleaved_offset(int row, int k, int K) {
    return (row >> 3) * (K >> 3) * 128 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2;
}

// GELU in its tanh form (Hendrycks & Gimpel 2016):
//   g(x) = x/2 (1 + tanh(u)),  u = sqrt(2/pi) (x + 0.044715 x^3),
// with the hardware tanh.approx.f32 (well below the BF16 rounding of the
// activations that follows), the same in inference and in training.
__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kGeluC = 0.7978845608028654f, kGeluA = 0.044715f;
// u = x (C + C A x^2), g = h + h t with h = x/2: six instructions (the
// epilogues apply it to every hidden activation).
__device__ __forceinline__ float gelu(float x) {
    const float t = tanh_hw(x * fmaf(kGeluC * kGeluA, x * x, kGeluC));
    const float h = 0.5f * x;
    return fmaf(h, t, h);
}
__device__ __forceinline__ float gelu_grad(float x) {
    const float t = tanh_hw(x * fmaf(kGeluC * kGeluA, x * x, kGeluC));
    return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * kGeluC * fmaf(3.f * kGeluA, x * x, 1.f);
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ---------------------------------------------------------------------------
// Packing: FP32 parameters -> BF16 tensor-core image (+ FP32 biases)
// ---------------------------------------------------------------------------
__global__ void k_mlp_pack(const float* __restrict__ prm, uint8_t* __restrict__ img) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    __nv_bfloat16* w1 = reinterpret_cast<__nv_bfloat16*>(img + kImgW1);
    __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(img + kImgW2);
    __nv_bfloat16* w3 = reinterpret_cast<__nv_bfloat16*>(img + kImgW3);
    float* bias = reinterpret_cast<float*>(img + kImgB);
    if (t < kMlpHid * kMlpInPad) {
        const int n = t / kMlpInPad, k = t % kMlpInPad;
        const float v = k < kMlpIn ? prm[kOffW1 + n * kMlpIn + k] : 0.f;
        w1[interleaved_offset(n, k, kMlpInPad) / 2] = __float2bfloat16_rn(v);
    }
    if (t < kMlpHid * kMlpHid) {
        const int n = t / kMlpHid, k = t % kMlpHid;
        w2[interleaved_offset(n, k, kMlpHid) / 2] = __float2bfloat16_rn(prm[kOffW2 + n * kMlpHid + k]);
    }
    if (t < kMlpOutPad * kMlpHid) {
        const int n = t / kMlpHid, k = t % kMlpHid;
        const float v = n < kMlpOut ? prm[kOffW3 + n * kMlpHid + k] : 0.f;
        w3[interleaved_offset(n, k, kMlpHid) / 2] = __float2bfloat16_rn(v);
    }
    if (t < kMlpHid) {
        bias[t] = prm[kOffB1 + t];
        bias[kMlpHid + t] = prm[kOffB2 + t];
    }
    if (t < kMlpOutPad) bias[2 * kMlpHid + t] = t < kMlpOut ? prm[kOffB3 + t] : 0.f;
}

// ---------------------------------------------------------------------------
// tcgen05 / bulk-copy / mbarrier helpers (inline PTX, sm_100a)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Bounded wait on phase `parity`; false when the bound ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int max_polls) {
    const uint32_t a = smem_u32(bar);
    for (int i = 0; i < max_polls; ++i) {
        uint32_t done = 0;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// The same for every thread of a CTA: false in all of them when the bound ran out in any, so that they go on together
// and whichever thread reports it has seen it.
__device__ __forceinline__ bool cta_wait(uint64_t* bar, uint32_t parity, int max_polls) {
    return __syncthreads_and(mbar_wait(bar, parity, max_polls)) != 0;
}
// 1-D bulk async copy global -> shared, completion counted on `bar` (16-byte
// aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// UMMA shared-memory descriptor, K-major, no swizzle: LBO = byte stride between
// the two 16-byte K chunks of one MMA, SBO = byte stride between 8-row groups.
__device__ __forceinline__ uint64_t umma_desc(const void* p, uint32_t lbo, uint32_t sbo) {
    const uint64_t addr = smem_u32(p);
    return ((addr >> 4) & 0x3FFFull) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) |
           (1ull << 46);   // version 1 (sm100), base offset 0, layout SWIZZLE_NONE
}
// Instruction descriptor, kind::f16: BF16 A and B (K-major), FP32 D, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// 32 lanes x 32-bit, 16 consecutive columns per thread.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Inference: one CTA per 128-row tile, grid-strided over tiles.
// ---------------------------------------------------------------------------
constexpr int kMlpThreads = 256;   // 8 warps: warp w serves TMEM lanes 32 (w % 4).. and hidden columns 32 (w / 4)..
constexpr int kTmemCols = 128;     // D1 cols [0,64), D2 [64,128), D3 [0,16): D1 has been read by then
constexpr int kMaxPolls = 1 << 22;

struct MlpSmem {
    alignas(128) uint8_t x[kTileBytes];                          // 128 x 16 bf16
    alignas(128) uint8_t w[kImgBytes];                           // weights + biases
    alignas(128) uint8_t h[kMlpTile * kMlpHid * 2];              // 128 x 64 bf16 (layer 2 and 3 A operand)
    alignas(8) uint64_t bar_load, bar_mma, bar_win;   // bar_win: the learned sweep's residual window
    uint32_t tmem_base;
    int stop;
};

// Dynamic shared memory of the kernels with tensor-core tiles: at least 48 KiB, so that at most four CTAs (4 x 128 TMEM
// columns) are resident per SM, of one kernel or of several, and tcgen05.alloc never waits.
constexpr size_t kMlpMinSmem = 48 * 1024;
inline size_t mlp_tc_smem_bytes() { return sizeof(MlpSmem) > kMlpMinSmem ? sizeof(MlpSmem) : kMlpMinSmem; }

// Bounded waits of one thread; the first wait that ran out is remembered so
// that it can be retried once before TMEM is released (no copy or MMA of the
// CTA is then left in flight).
struct WaitState {
    uint64_t* fail_bar = nullptr;
    uint32_t fail_par = 0;
};
__device__ __forceinline__ bool wait_bar(WaitState& ws, uint64_t* bar, uint32_t par) {
    const bool done = mbar_wait(bar, par, kMaxPolls);
    if (!done && !ws.fail_bar) {
        ws.fail_bar = bar;
        ws.fail_par = par;
    }
    return done;
}

// CTA prologue: barriers, TMEM (128 columns, warp 0) and the weight image.
// With wait_weights = false the copy is left in flight (the caller overlaps it
// with other work and calls mlp_wait_weights before the first MMA).
__device__ __forceinline__ uint32_t mlp_cta_setup(MlpSmem& S, const uint8_t* img, WaitState& ws, uint32_t& ph_load,
                                                  int32_t* err, bool wait_weights = true) {
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(&S.bar_load, 1);
        mbar_init(&S.bar_mma, 1);
        mbar_init(&S.bar_win, 1);
        S.stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&S.bar_load, kImgBytes);
        bulk_g2s(S.w, img, kImgBytes, &S.bar_load);
    }
    if (wait_weights) {
        if (!wait_bar(ws, &S.bar_load, ph_load)) {
            S.stop = 1;
            if (err) atomicExch(err, 1);
        }
        ph_load ^= 1;
    }
    return S.tmem_base;
}

// Completes a weight copy left in flight by mlp_cta_setup(..., false).
__device__ __forceinline__ bool mlp_wait_weights(MlpSmem& S, WaitState& ws, uint32_t& ph_load, int32_t* err) {
    const bool ok = wait_bar(ws, &S.bar_load, ph_load);
    ph_load ^= 1;
    if (!ok) {
        S.stop = 1;
        if (err) atomicExch(err, 1);
    }
    return ok;
}

// CTA epilogue: retry a timed-out wait once, then release TMEM.
__device__ __forceinline__ void mlp_cta_teardown(MlpSmem& S, uint32_t tmem, WaitState& ws) {
    if (ws.fail_bar) mbar_wait(ws.fail_bar, ws.fail_par, kMaxPolls);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if ((threadIdx.x >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// Hidden layer epilogue: gelu(D + bias) of this warp's half of the 64 columns
// (c0 = 0 or 32) of this thread's row, from TMEM -> BF16 into S.h (K-major
// interleaved, K = 64).
__device__ __forceinline__ void mlp_hidden_epilogue(MlpSmem& S, uint32_t taddr, const float* bias, int row_in_tile,
                                                    int c0) {
    // both 16-column loads in flight before the one wait
    static_assert(kMlpHid / 2 == 32, "a warp's half of the hidden columns is two 16-column loads");
    float v[2][16];
    tmem_ld16(taddr + c0, v[0]);
    tmem_ld16(taddr + c0 + 16, v[1]);
    tmem_wait_ld();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = c0 + 16 * h;
        uint32_t packed[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const __nv_bfloat162 two = __floats2bfloat162_rn(gelu(v[h][2 * i] + bias[c + 2 * i]),
                                                             gelu(v[h][2 * i + 1] + bias[c + 2 * i + 1]));
            packed[i] = *reinterpret_cast<const uint32_t*>(&two);
        }
        uint8_t* base = S.h + interleaved_offset(row_in_tile, c, kMlpHid);
        *reinterpret_cast<uint4*>(base) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        *reinterpret_cast<uint4*>(base + 128) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    }
}

// The three layers on the feature tile in S.x (which the caller has made
// visible to the async proxy and synchronised); y receives this thread's row.
// Returns false when a wait ran out.
__device__ __forceinline__ bool mlp_tile_layers(MlpSmem& S, uint32_t tmem, uint32_t& ph_mma, WaitState& ws, bool ok,
                                                float (&y)[3]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = warp & 3, c0 = (warp >> 2) * (kMlpHid / 2);
    const int row_in_tile = grp * 32 + lane;
    const uint32_t lane_base = (uint32_t)(grp * 32) << 16;
    const float* bias = reinterpret_cast<const float*>(S.w + kImgB);
    const uint32_t id64 = umma_idesc_bf16(kMlpTile, kMlpHid), id16 = umma_idesc_bf16(kMlpTile, kMlpOutPad);
    // layer 1: D1 = X W1^T (K = 16: one MMA)
    tc_fence_after();
    if (threadIdx.x == 0 && ok) {
        umma_bf16(tmem + 0, umma_desc(S.x, 128, 256), umma_desc(S.w + kImgW1, 128, 256), id64, 0);
        umma_commit(&S.bar_mma);
    }
    ok = ok && wait_bar(ws, &S.bar_mma, ph_mma);
    ph_mma ^= 1;
    tc_fence_after();
    mlp_hidden_epilogue(S, tmem + lane_base + 0, bias, row_in_tile, c0);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // layer 2: D2 = H1 W2^T (K = 64: four MMAs)
    if (threadIdx.x == 0 && ok) {
#pragma unroll
        for (int k = 0; k < kMlpHid / 16; ++k)
            umma_bf16(tmem + 64, umma_desc(S.h + k * 256, 128, 1024), umma_desc(S.w + kImgW2 + k * 256, 128, 1024), id64,
                      k > 0 ? 1u : 0u);
        umma_commit(&S.bar_mma);
    }
    ok = ok && wait_bar(ws, &S.bar_mma, ph_mma);
    ph_mma ^= 1;
    tc_fence_after();
    // H2 overwrites H1: layer 2 has finished reading it
    mlp_hidden_epilogue(S, tmem + lane_base + 64, bias + kMlpHid, row_in_tile, c0);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // layer 3: D3 = H2 W3^T (N = 16, 3 used)
    if (threadIdx.x == 0 && ok) {
#pragma unroll
        for (int k = 0; k < kMlpHid / 16; ++k)
            umma_bf16(tmem, umma_desc(S.h + k * 256, 128, 1024), umma_desc(S.w + kImgW3 + k * 256, 128, 1024),
                      id16, k > 0 ? 1u : 0u);
        umma_commit(&S.bar_mma);
    }
    ok = ok && wait_bar(ws, &S.bar_mma, ph_mma);
    ph_mma ^= 1;
    tc_fence_after();
    float v[16];
    tmem_ld16(tmem + lane_base, v);   // every warp (the .sync.aligned load is warp-wide); warps 0-3 use it
    tmem_wait_ld();
    tc_fence_before();
    y[0] = v[0] + bias[2 * kMlpHid];
    y[1] = v[1] + bias[2 * kMlpHid + 1];
    y[2] = v[2] + bias[2 * kMlpHid + 2];
    return ok;
}

// One row of FP32 features into the BF16 operand tile (K padded 9 -> 16 with zeros).
__device__ __forceinline__ void mlp_store_features(uint8_t* tile, int row_in_tile, const float (&f)[kMlpIn]) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float lo = 2 * i < kMlpIn ? f[2 * i] : 0.f;
        const float hi = 2 * i + 1 < kMlpIn ? f[2 * i + 1] : 0.f;
        const __nv_bfloat162 two = __floats2bfloat162_rn(lo, hi);
        w[i] = *reinterpret_cast<const uint32_t*>(&two);
    }
    uint8_t* base = tile + interleaved_offset(row_in_tile, 0, kMlpInPad);
    *reinterpret_cast<uint4*>(base) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(base + 128) = make_uint4(w[4], w[5], w[6], w[7]);
}

// Inference on row-major features x[n][9], outputs y[n][3]: one CTA per 128-row tile, grid-strided; a thread per row
// rounds the row's features straight into the operand tile.  err: set to 1 when a bounded wait ran out; the kernel
// then stops.
__global__ void __launch_bounds__(kMlpThreads) k_mlp_tc(int n, int ntiles, const float* __restrict__ x,
                                                        const uint8_t* __restrict__ img, float* __restrict__ y,
                                                        int32_t* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    MlpSmem& S = *reinterpret_cast<MlpSmem*>(smem_raw);
    WaitState ws;
    uint32_t ph_load = 0, ph_mma = 0;
    const uint32_t tmem = mlp_cta_setup(S, img, ws, ph_load, err);
    const int row_in_tile = threadIdx.x;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        __syncthreads();
        if (S.stop) break;
        const int row = tile * kMlpTile + row_in_tile;
        if (row_in_tile < kMlpTile) {
            float f[kMlpIn];
#pragma unroll
            for (int k = 0; k < kMlpIn; ++k) f[k] = row < n ? x[(size_t)row * kMlpIn + k] : 0.f;
            mlp_store_features(S.x, row_in_tile, f);
        }
        fence_async_shared();
        tc_fence_before();
        __syncthreads();
        float out[3];
        const bool ok = mlp_tile_layers(S, tmem, ph_mma, ws, true, out);
        if (!ok) {
            S.stop = 1;
            if (err) atomicExch(err, 1);
        }
        if (ok && row_in_tile < kMlpTile && row < n) {
            y[3 * (size_t)row] = out[0];
            y[3 * (size_t)row + 1] = out[1];
            y[3 * (size_t)row + 2] = out[2];
        }
    }
    mlp_cta_teardown(S, tmem, ws);
}

// ---------------------------------------------------------------------------
// Training: forward + backward, FP32 math with the same BF16 rounding of the
// weights and activations as the tensor-core forward (straight-through in the
// backward).  Loss = mean over samples and the 3 outputs of (y - t)^2.
//
// A step is a chain of two launches.  k_mlp_fwd_bwd takes 32 samples per CTA (a
// sample per lane, 4 hidden units per warp) and leaves the rows that the weight
// gradients multiply -- features, dZ1, H1, dZ2, H2, dY -- in global scratch, a
// row per unit over all samples.  k_mlp_grad gives each CTA a tile of
// parameters: their rows arrive in shared memory by bulk copies, a thread forms
// the dot products of one 128-sample block, and the blocks are added in
// ascending order, without atomics (deterministic); the same thread then takes
// the Adam step.  Both kernels fill the chip at 4,096 samples (128 and 127 CTAs
// of 148 SMs); one CTA per 128 samples for everything, as before, left 116 SMs
// idle: 100 steps on 200,000 pairs took 10.1 ms with its four small launches, and
// take 2.65 ms (the upload of the pairs included).  Every sum runs in the order of
// that form: the same bits.
// ---------------------------------------------------------------------------
constexpr int kTrainThreads = 512;            // 16 warps of 4 hidden units each
constexpr int kTrainUnits = 4;
constexpr int kTrainSamples = 32;             // per CTA
constexpr int kGradBlock = 128;               // samples of one dot product
constexpr int kGradLd = kGradBlock + 4;       // its place in a scratch row: 16-byte reads of 8 blocks miss no bank
constexpr int kTrainChunk = 8192;             // samples of one launch pair at most (9 MB of scratch)
// scratch rows
constexpr int kActX = 0, kActZ1 = kActX + kMlpIn, kActH1 = kActZ1 + kMlpHid, kActZ2 = kActH1 + kMlpHid,
              kActH2 = kActZ2 + kMlpHid, kActY = kActH2 + kMlpHid, kActRows = kActY + kMlpOut;

__host__ __device__ inline int train_blocks(int n) { return (n + kGradBlock - 1) / kGradBlock; }

struct TrainSmem {
    float w1[kMlpIn][kMlpHid];     // [k][j]
    float w2t[kMlpHid][kMlpHid + 4];   // [k][j], forward
    float w2[kMlpHid][kMlpHid + 4];    // [j][k], backward
    float w3[kMlpOut][kMlpHid];
    float b1[kMlpHid], b2[kMlpHid], b3[kMlpOut + 1];
    float x[kMlpIn][kTrainSamples];
    float h1[kMlpHid][kTrainSamples], h2[kMlpHid][kTrainSamples], z2[kMlpHid][kTrainSamples];
    float d[kMlpOut][kTrainSamples], dy[kMlpOut][kTrainSamples];
};

// Row of sample s of a minibatch: s itself, or uniform in [0, n) from a counter-based hash (splitmix64).
struct SampleOf {
    int sampled, first, n;
    uint64_t seed, step;
    __device__ __forceinline__ int operator()(int s) const {
        if (!sampled) return first + s;
        uint64_t z = seed + (step * 0x9E3779B97F4A7C15ull) + (uint64_t)(first + s) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (int)(z % (uint64_t)n);
    }
};

// nb samples of this launch; ld: floats of a scratch row.  lsum[s]: the sample's squared error.
__global__ void __launch_bounds__(kTrainThreads) k_mlp_fwd_bwd(int nb, SampleOf sample, const float* __restrict__ X,
                                                               const float* __restrict__ T, const float* __restrict__ prm,
                                                               float* __restrict__ act, int ld, float* __restrict__ lsum,
                                                               float inv_count) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(16) unsigned char train_smem[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(train_smem);
    const int s = threadIdx.x & 31, warp = threadIdx.x >> 5, j0 = kTrainUnits * warp;
    const int gs = blockIdx.x * kTrainSamples + s;
    const bool valid = gs < nb;
    // the samples are not written by any kernel of a training run: read before the wait
    const int row = valid ? sample(gs) : 0;
    for (int k = warp; k < kMlpIn; k += kTrainThreads / 32) S.x[k][s] = valid ? bf16r(X[(size_t)row * kMlpIn + k]) : 0.f;
    const float target = valid && warp < kMlpOut ? T[(size_t)row * kMlpOut + warp] : 0.f;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // weights, BF16-rounded, and exact biases
    {   // a thread per row of 64 and 4 columns at a time: the stores to both copies miss no bank
        static_assert(kOffW2 % 4 == 0 && kTrainThreads == 8 * kMlpHid, "16-byte reads, 8 columns a thread");
        const int j = threadIdx.x % kMlpHid, k0 = threadIdx.x / kMlpHid * 8;
        const float4* from = reinterpret_cast<const float4*>(prm + kOffW2 + j * kMlpHid + k0);
        const float4 q[2] = {from[0], from[1]};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 w = make_float4(bf16r(q[h].x), bf16r(q[h].y), bf16r(q[h].z), bf16r(q[h].w));
            const int k = k0 + 4 * h;
            *reinterpret_cast<float4*>(&S.w2[j][k]) = w;
            S.w2t[k][j] = w.x;
            S.w2t[k + 1][j] = w.y;
            S.w2t[k + 2][j] = w.z;
            S.w2t[k + 3][j] = w.w;
        }
    }
    for (int q = threadIdx.x; q < kMlpHid * kMlpIn; q += kTrainThreads) S.w1[q % kMlpIn][q / kMlpIn] = bf16r(prm[kOffW1 + q]);
    if (threadIdx.x < kMlpOut * kMlpHid) S.w3[threadIdx.x / kMlpHid][threadIdx.x % kMlpHid] = bf16r(prm[kOffW3 + threadIdx.x]);
    if (threadIdx.x < kMlpHid) {
        S.b1[threadIdx.x] = prm[kOffB1 + threadIdx.x];
        S.b2[threadIdx.x] = prm[kOffB2 + threadIdx.x];
    }
    if (threadIdx.x < kMlpOut) S.b3[threadIdx.x] = prm[kOffB3 + threadIdx.x];
    __syncthreads();
    auto row_units = [](const float* p, float (&w)[kTrainUnits]) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    };
    // place of this sample in the scratch rows
    float* at = act + (size_t)(gs / kGradBlock) * kGradLd + gs % kGradBlock;
    for (int k = warp; k < kMlpIn; k += kTrainThreads / 32) at[(size_t)(kActX + k) * ld] = S.x[k][s];
    // ---- forward
    float z1[kTrainUnits], z2[kTrainUnits], w[kTrainUnits];
    row_units(S.b1 + j0, z1);
#pragma unroll
    for (int k = 0; k < kMlpIn; ++k) {
        row_units(&S.w1[k][j0], w);
        const float x = S.x[k][s];
#pragma unroll
        for (int u = 0; u < kTrainUnits; ++u) z1[u] = fmaf(w[u], x, z1[u]);
    }
#pragma unroll
    for (int u = 0; u < kTrainUnits; ++u) {
        const float h = bf16r(gelu(z1[u]));
        S.h1[j0 + u][s] = h;
        at[(size_t)(kActH1 + j0 + u) * ld] = h;
    }
    __syncthreads();
    row_units(S.b2 + j0, z2);
#pragma unroll 8
    for (int k = 0; k < kMlpHid; ++k) {
        row_units(&S.w2t[k][j0], w);
        const float h = S.h1[k][s];
#pragma unroll
        for (int u = 0; u < kTrainUnits; ++u) z2[u] = fmaf(w[u], h, z2[u]);
    }
#pragma unroll
    for (int u = 0; u < kTrainUnits; ++u) {
        const float h = bf16r(gelu(z2[u]));
        S.h2[j0 + u][s] = h;
        at[(size_t)(kActH2 + j0 + u) * ld] = h;
    }
    __syncthreads();
    if (warp < kMlpOut) {
        float a = S.b3[warp];
#pragma unroll 16
        for (int k = 0; k < kMlpHid; ++k) a = fmaf(S.w3[warp][k], S.h2[k][s], a);
        const float d = valid ? a - target : 0.f;
        const float dy = 2.f * d * inv_count;
        S.d[warp][s] = d;
        S.dy[warp][s] = dy;
        at[(size_t)(kActY + warp) * ld] = dy;
    }
    __syncthreads();
    if (warp == 0) {
        float loss = 0.f;
#pragma unroll
        for (int o = 0; o < kMlpOut; ++o) {
            const float d = S.d[o][s];
            loss += d * d;
        }
        lsum[gs] = loss;
    }
    // ---- backward through layers 3 and 2
#pragma unroll
    for (int u = 0; u < kTrainUnits; ++u) {
        float a = 0.f;
#pragma unroll
        for (int o = 0; o < kMlpOut; ++o) a = fmaf(S.dy[o][s], S.w3[o][j0 + u], a);
        const float z = a * gelu_grad(z2[u]);
        S.z2[j0 + u][s] = z;
        at[(size_t)(kActZ2 + j0 + u) * ld] = z;
    }
    __syncthreads();
    float a1[kTrainUnits];
#pragma unroll
    for (int u = 0; u < kTrainUnits; ++u) a1[u] = 0.f;
#pragma unroll 8
    for (int j = 0; j < kMlpHid; ++j) {
        row_units(&S.w2[j][j0], w);
        const float z = S.z2[j][s];
#pragma unroll
        for (int u = 0; u < kTrainUnits; ++u) a1[u] = fmaf(z, w[u], a1[u]);
    }
#pragma unroll
    for (int u = 0; u < kTrainUnits; ++u) at[(size_t)(kActZ1 + j0 + u) * ld] = a1[u] * gelu_grad(z1[u]);
}

// Adam (Kingma & Ba 2015) on one FP32 master parameter.
struct AdamStep {
    float lr, b1, b2, eps, bc1, bc2;
};
__device__ __forceinline__ void adam(float gq, float* prm, float* m, float* v, int q, const AdamStep& A) {
    const float mq = A.b1 * m[q] + (1.f - A.b1) * gq;
    const float vq = A.b2 * v[q] + (1.f - A.b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    prm[q] -= A.lr * (mq / A.bc1) / (sqrtf(vq / A.bc2) + A.eps);
}

// Parameter tiles: rows u of one scratch group against rows v of another, 13 rows of shared memory at most.
constexpr int kGradGroups = 32;   // blocks of 128 samples in shared memory at a time, a lane each
constexpr int kGradThreads = 64;  // two halves of the tile, 32 blocks each
constexpr int kGradRows = 13;
constexpr int kTiles2 = 8 * 13;   // W2: 8 x 5 parameters of dZ2 x H1
constexpr int kTiles1 = 16;       // W1: 4 x 9 of dZ1 x features
constexpr int kTiles3 = 7;        // W3: 3 x 10 of dY x H2
constexpr int kGradTiles = kTiles2 + kTiles1 + kTiles3;
constexpr int kGradParams = 48;   // most parameters of a tile, biases included

struct GradSmem {
    alignas(128) float row[kGradRows][kGradGroups * kGradLd];
    float part[kGradParams][kGradGroups + 1];
    float loss[kGradGroups];
    uint64_t bar;
};

// Dot products of MU rows u and MV rows v over one block of 128 samples, and the sums of the rows u.
template <int MU, int MV>
__device__ __forceinline__ void grad_dots(const float* const (&u)[MU], const float* const (&v)[MV], float (&dot)[MU][MV],
                                          float (&sum)[MU]) {
#pragma unroll
    for (int i = 0; i < MU; ++i) {
        sum[i] = 0.f;
#pragma unroll
        for (int j = 0; j < MV; ++j) dot[i][j] = 0.f;
    }
#pragma unroll 2
    for (int t = 0; t < kGradBlock; t += 4) {
        float a[MU][4], b[MV][4];
#pragma unroll
        for (int i = 0; i < MU; ++i) {
            const float4 q = *reinterpret_cast<const float4*>(u[i] + t);
            a[i][0] = q.x; a[i][1] = q.y; a[i][2] = q.z; a[i][3] = q.w;
        }
#pragma unroll
        for (int j = 0; j < MV; ++j) {
            const float4 q = *reinterpret_cast<const float4*>(v[j] + t);
            b[j][0] = q.x; b[j][1] = q.y; b[j][2] = q.z; b[j][3] = q.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < MU; ++i) {
                sum[i] += a[i][k];
#pragma unroll
                for (int j = 0; j < MV; ++j) dot[i][j] = fmaf(a[i][k], b[j][k], dot[i][j]);
            }
    }
}

// One thread's share of a tile: rows u0.. and v0.. of S.row, block `lane`; parameter (i, j) of the tile's U x V goes to
// part[i * V + j], the sums of the rows u to part[U * V + i].
template <int MU, int MV>
__device__ __forceinline__ void grad_tile(GradSmem& S, int lane, int u0, int v0, int U, int V, int i0, int j0, bool sums) {
    const float *u[MU], *v[MV];
#pragma unroll
    for (int i = 0; i < MU; ++i) u[i] = S.row[u0 + i] + lane * kGradLd;
#pragma unroll
    for (int j = 0; j < MV; ++j) v[j] = S.row[v0 + j] + lane * kGradLd;
    float dot[MU][MV], sum[MU];
    grad_dots<MU, MV>(u, v, dot, sum);
#pragma unroll
    for (int i = 0; i < MU; ++i) {
#pragma unroll
        for (int j = 0; j < MV; ++j)
            if (j0 + j < V) S.part[(i0 + i) * V + j0 + j][lane] = dot[i][j];   // else a row past a narrower tile
        if (sums) S.part[U * V + i0 + i][lane] = sum[i];
    }
}

// Gradient of a launch's nblk blocks of 128 samples, tile blockIdx.x.  acc: the sums of the launches before it (grad,
// loss), else 0.  final: inv_count scales the loss, and with prm the Adam step is taken; else the sums stay in grad.
__global__ void __launch_bounds__(kGradThreads) k_mlp_grad(int nblk, const float* __restrict__ act, int ld,
                                                           const float* __restrict__ lsum, int acc, int final, float inv_count,
                                                           float* __restrict__ grad, float* __restrict__ loss,
                                                           float* __restrict__ loss_out, float* __restrict__ prm,
                                                           float* __restrict__ m, float* __restrict__ v, AdamStep A,
                                                           int32_t* __restrict__ err) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(128) unsigned char grad_smem[];
    GradSmem& S = *reinterpret_cast<GradSmem*>(grad_smem);
    const int lane = threadIdx.x & 31, half = threadIdx.x >> 5;
    // the tile: U rows from u_at against V rows from v_at; its first parameter and row stride; its biases
    int U, V, u_at, v_at, q0, stride, bias = -1;
    int tile = blockIdx.x;
    const int kind = tile < kTiles2 ? 2 : tile < kTiles2 + kTiles1 ? 1 : 3;
    if (kind == 2) {
        const int r = tile / 13, c = tile % 13;
        U = 8;
        V = min(5, kMlpHid - 5 * c);
        u_at = kActZ2 + 8 * r;
        v_at = kActH1 + 5 * c;
        q0 = kOffW2 + 8 * r * kMlpHid + 5 * c;
        stride = kMlpHid;
        if (c == 0) bias = kOffB2 + 8 * r;
    } else if (kind == 1) {
        tile -= kTiles2;
        U = 4;
        V = kMlpIn;
        u_at = kActZ1 + 4 * tile;
        v_at = kActX;
        q0 = kOffW1 + 4 * tile * kMlpIn;
        stride = kMlpIn;
        bias = kOffB1 + 4 * tile;
    } else {
        tile -= kTiles2 + kTiles1;
        U = kMlpOut;
        V = min(10, kMlpHid - 10 * tile);
        u_at = kActY;
        v_at = kActH2 + 10 * tile;
        q0 = kOffW3 + 10 * tile;
        stride = kMlpHid;
        if (tile == 0) bias = kOffB3;
    }
    const int many = U * V + (bias >= 0 ? U : 0);   // parameters of the tile
    auto param = [&](int p) { return p < U * V ? q0 + p / V * stride + p % V : bias + p - U * V; };
    if (threadIdx.x == 0) {
        mbar_init(&S.bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float g = 0.f, l = 0.f;   // this thread's parameter; thread 0 of the first tile: the loss
    if (acc && threadIdx.x < many) g = grad[param(threadIdx.x)];
    const bool loss_tile = blockIdx.x == gridDim.x - 1;   // the smallest
    if (acc && loss_tile && threadIdx.x == 0) l = *loss;
    bool ok = true;
    uint32_t phase = 0;
    for (int b0 = 0; b0 < nblk && ok; b0 += kGradGroups, phase ^= 1) {
        const int nb = min(kGradGroups, nblk - b0);
        if (threadIdx.x == 0) {
            mbar_expect_tx(&S.bar, (uint32_t)((U + V) * nb * kGradLd * 4));
            for (int r = 0; r < U + V; ++r)
                bulk_g2s(S.row[r], act + (size_t)(r < U ? u_at + r : v_at + r - U) * ld + (size_t)b0 * kGradLd,
                         (uint32_t)(nb * kGradLd * 4), &S.bar);
        }
        if (loss_tile && half == 1 && lane < nb) {   // the blocks' losses, in sample order
            const float4* p = reinterpret_cast<const float4*>(lsum + (size_t)(b0 + lane) * kGradBlock);
            float t = 0.f;
#pragma unroll 8
            for (int i = 0; i < kGradBlock / 4; ++i) {
                const float4 q = __ldg(p + i);
                t += q.x;
                t += q.y;
                t += q.z;
                t += q.w;
            }
            S.loss[lane] = t;
        }
        ok = cta_wait(&S.bar, phase, kMaxPolls);
        if (ok && lane < nb) {
            if (kind == 2)
                grad_tile<4, 5>(S, lane, 4 * half, U, U, V, 4 * half, 0, bias >= 0);
            else if (kind == 1)
                grad_tile<2, 9>(S, lane, 2 * half, U, U, V, 2 * half, 0, true);
            else
                grad_tile<3, 5>(S, lane, 0, U + 5 * half, U, V, 0, 5 * half, bias >= 0 && half == 0);
        }
        __syncthreads();
        if (ok && threadIdx.x < many)
            for (int b = 0; b < nb; ++b) g += S.part[threadIdx.x][b];
        if (loss_tile && threadIdx.x == 0)
            for (int b = 0; b < nb; ++b) l += S.loss[b];
        __syncthreads();
    }
    if (!ok) {   // report, and leave no copy in flight
        if (threadIdx.x == 0) atomicExch(err, 1);
        mbar_wait(&S.bar, phase ^ 1, kMaxPolls);
        return;
    }
    if (threadIdx.x < many) {
        const int q = param(threadIdx.x);
        if (final && prm)
            adam(g, prm, m, v, q, A);
        else
            grad[q] = g;
    }
    if (loss_tile && threadIdx.x == 0) {
        if (final) l *= inv_count;
        *loss = l;
        if (final && loss_out) *loss_out = l;
    }
}

}  // namespace
}  // namespace mgsb
