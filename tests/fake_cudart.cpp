// A stand-in for the CUDA runtime under the host code of the solvers, for tests without a GPU: memory is host memory,
// copies are copies, a kernel launch is written down (name, grid, block, shared memory, cluster, cooperative) and does
// nothing else.  A launch can be refused by kernel name, as the runtime refuses one that does not fit the device.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string kernel;
    unsigned grid, block, cluster, cooperative;
    size_t smem;
};
std::map<const void*, std::string> kernels;
std::vector<Launch> launches;
std::string refused;
long counts[6];   // captures, graph launches, stream synchronisations, bytes copied to the device, pinned allocations, bytes
                  // of device memory
cudaError_t last = cudaSuccess;
char token[8];    // what handles point at

cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem, unsigned cluster, unsigned cooperative) {
    const std::string& name = kernels[f];
    if (!refused.empty() && name.find(refused) != std::string::npos) return last = cudaErrorCooperativeLaunchTooLarge;
    launches.push_back({name, g.x, b.x, cluster, cooperative, smem});
    return cudaSuccess;
}
template <typename T>
cudaError_t handle(T* out) {
    *out = reinterpret_cast<T>(token);
    return cudaSuccess;
}
cudaError_t host_malloc(void** p, size_t n) {
    const size_t size = (n + 255) / 256 * 256 + 256;
    *p = aligned_alloc(256, size);
    return *p ? memset(*p, 0, size), cudaSuccess : cudaErrorMemoryAllocation;
}
thread_local struct { dim3 g, b; size_t smem; void* s; } config;
}  // namespace

extern "C" {
// ---- what the tests see
void fake_reset() {
    launches.clear();
    refused.clear();
    memset(counts, 0, sizeof counts);
}
void fake_refuse(const char* name) { refused = name; }
long fake_count(int what) { return counts[what]; }
int fake_launches() { return (int)launches.size(); }
int fake_launch(int k, char* name, int cap, unsigned long long out[5]) {
    const Launch& l = launches[(size_t)k];
    std::snprintf(name, (size_t)cap, "%s", l.kernel.c_str());
    out[0] = l.grid, out[1] = l.block, out[2] = l.cluster, out[3] = l.cooperative, out[4] = l.smem;
    return 0;
}

// ---- what nvcc's host code calls
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(token); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) {
    kernels[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) {
    config = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = config.g, *b = config.b, *smem = config.smem;
    *static_cast<void**>(s) = config.s;
    return cudaSuccess;
}

// ---- the runtime
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
    return launch(f, g, b, smem, 0, 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    unsigned cluster = 0, cooperative = 0;
    for (unsigned k = 0; k < c->numAttrs; ++k) {
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[k].val.clusterDim.x;
        if (c->attrs[k].id == cudaLaunchAttributeCooperative) cooperative = (unsigned)c->attrs[k].val.cooperative;
    }
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, cluster, cooperative);
}
cudaError_t cudaMalloc(void** p, size_t n) { return counts[5] += (long)n, host_malloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return ++counts[4], host_malloc(p, n); }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    if (k == cudaMemcpyHostToDevice) counts[3] += (long)n;
    return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k) {
    for (size_t r = 0; r < h; ++r) cudaMemcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w, k);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448
         : a == cudaDevAttrCooperativeLaunch ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { return *n = 1, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    return *n = 1, cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return ++counts[0], cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return handle(e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return ++counts[1], cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return ++counts[2], cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    return last = cudaSuccess, e;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
// conditional nodes, symbols and driver entry points: not there
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams*) {
    return cudaErrorNotSupported;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned) {
    return cudaErrorNotSupported;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                          cudaStreamCaptureMode) {
    return cudaErrorNotSupported;
}
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus*, unsigned long long*, cudaGraph_t*,
                                        const cudaGraphNode_t**, size_t*) {
    return cudaErrorNotSupported;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { return *s = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, size_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorNotSupported; }
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) {
    return cudaErrorNotSupported;
}
}
