// A CUDA runtime without a device, linked with the library's own objects in place of libcudart so that its host code (which
// kernel, which grid, what happens when a call fails) runs on a CPU. Device addresses are numbers that nothing reads. Every
// launch is checked against the grid limits of compute capability 10.0 and written down; allocations above a limit and a chosen
// number of occupancy queries fail, and a failed call is the thread's last error until cudaGetLastError, as in the real runtime.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string> kernels;
std::string log_text;
size_t pool_limit = SIZE_MAX;
int occupancy_failures = 0;
int encoded = 0;  // tensor maps since fake_reset
cudaError_t last = cudaSuccess;
uintptr_t next_address = 1ull << 40;

cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
void* address(size_t bytes) {
    const uintptr_t p = next_address;
    next_address += (bytes + 4095) & ~(size_t)4095;
    return reinterpret_cast<void*>(p);
}
cudaError_t launch(const void* func, dim3 g, dim3 b, size_t smem, unsigned cluster, int ahead = 0) {
    if (g.x == 0 || g.y == 0 || g.z == 0 || g.x > 0x7fffffffu || g.y > 65535u || g.z > 65535u || b.x * b.y * b.z > 1024u)
        return result(cudaErrorInvalidConfiguration);
    char line[512];
    snprintf(line, sizeof(line), "%s grid %u %u %u block %u smem %zu ahead %d cluster %u\n", kernels[func].c_str(), g.x, g.y, g.z, b.x * b.y * b.z, smem, ahead, cluster);
    log_text += line;
    return cudaSuccess;
}
CUresult encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    ++encoded;
    memset(m, 0, sizeof(*m));
    return CUDA_SUCCESS;
}
}  // namespace

extern "C" {
// ---- what the tests set and read
void fake_reset(void) {
    log_text.clear();
    pool_limit = SIZE_MAX;
    occupancy_failures = 0;
    encoded = 0;
    last = cudaSuccess;
}
void fake_pool_limit(size_t bytes) { pool_limit = bytes; }
void fake_fail_occupancy(int times) { occupancy_failures = times; }
int fake_encoded(void) { return encoded; }
const char* fake_launches(void) { return log_text.c_str(); }

// ---- the runtime
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { kernels[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static thread_local struct { dim3 g, b; size_t smem; void* s; } pushed;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) { pushed = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = pushed.g; *b = pushed.b; *smem = pushed.smem; *static_cast<void**>(s) = pushed.s;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) { return launch(f, g, b, smem, 1); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    unsigned cluster = 1;
    int ahead = 0;  // of the end of the kernel before
    for (unsigned i = 0; i < c->numAttrs; ++i) {
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
        if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) ahead = c->attrs[i].val.programmaticStreamSerializationAllowed;
    }
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, cluster, ahead);
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaErrorInvalidConfiguration ? "invalid configuration argument" : "error"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 10; return cudaSuccess; }  // (the compute capability's major is all that is asked)
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
// clusters of 2..8 CTAs of one per SM that a B200 holds at once, as its own runtime answers
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    static const int held[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    if (occupancy_failures > 0) { --occupancy_failures; return result(cudaErrorUnknown); }
    *n = held[c->attrs[0].val.clusterDim.x];
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = address(1); return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *fn = reinterpret_cast<void*>(encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { *p = address(n); return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { *p = address(n); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    if (n > pool_limit) return result(cudaErrorMemoryAllocation);
    *p = address(n);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = reinterpret_cast<cudaMemPool_t>(address(1)); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return result(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return result(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return result(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return result(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(address(1)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
}
