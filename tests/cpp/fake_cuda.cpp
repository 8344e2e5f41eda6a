// fake_cuda.cpp - TEST INFRASTRUCTURE: a CUDA runtime without a device, linked
// with the library's own object files, so that the host side of an upload runs
// on a machine without a GPU and any of its allocations can be made to fail.
// Device memory is host memory, copies and fills happen at once, kernels do
// nothing (but for the values below that steer the host's way); what counts is
// recorded: live bytes, allocations, and whether a stream has had work since it
// was last waited for.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

#include "../../shiro_gb300/csrc/pool.h"

namespace {

std::map<void*, size_t> gLive;
std::map<const void*, std::string> gKernels;
std::set<cudaStream_t> gBusy;
size_t gLiveBytes = 0, gCap = ~size_t(0);
long gMallocs = 0, gFailFrom = -1;
cudaError_t gLast = cudaSuccess;
struct Call {
    dim3 grid, block;
    size_t shared;
    cudaStream_t stream;
} gCall;

cudaError_t record(cudaError_t e) {
    if (e != cudaSuccess) gLast = e;
    return e;
}

void hook(const std::string& name, void** args) {
    const auto has = [&](const char* s) { return name.find(s) != std::string::npos; };
    if (has("k_flat_verts")) {  // the largest coordinate: too large for the wide BVH
        const float mag = 2.0e9f;
        std::memcpy(*static_cast<void**>(args[3]), &mag, sizeof(mag));
    } else if (has("k_env_mass")) {  // weights: sum and largest
        const unsigned long long stats[2] = {1000, 10};
        std::memcpy(*static_cast<void**>(args[6]), stats, sizeof(stats));
    }
}

}  // namespace

extern "C" {

// ---- the tests' side -------------------------------------------------------
void fake_reset(long failFrom, size_t cap) {
    gMallocs = 0;
    gFailFrom = failFrom;
    gCap = cap;
}
long fake_mallocs() { return gMallocs; }
size_t fake_live_bytes() { return gLiveBytes; }
int fake_busy_streams() { return static_cast<int>(gBusy.size()); }

void* fake_pool_new() { return new shiro_gpu::DevicePool(); }
void fake_pool_delete(void* p) { delete static_cast<shiro_gpu::DevicePool*>(p); }
void* fake_pool_get(void* p, size_t bytes) {
    void* out = nullptr;
    return static_cast<shiro_gpu::DevicePool*>(p)->get(&out, bytes) == cudaSuccess ? out : nullptr;
}
void fake_pool_put(void* p, void* block) { static_cast<shiro_gpu::DevicePool*>(p)->put(block); }

// ---- what nvcc's host code calls --------------------------------------------
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    gKernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
    gCall = Call{grid, block, shared, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream) {
    *grid = gCall.grid;
    *block = gCall.block;
    *shared = gCall.shared;
    *static_cast<cudaStream_t*>(stream) = gCall.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* out, const void* host) {
    *out = reinterpret_cast<cudaKernel_t>(const_cast<void*>(host));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t, cudaStream_t stream) {
    gBusy.insert(stream);
    hook(gKernels[reinterpret_cast<const void*>(k)], args);
    return cudaSuccess;
}

// ---- the runtime API ---------------------------------------------------------
cudaError_t cudaMalloc(void** out, size_t bytes) {
    const long n = ++gMallocs;
    *out = nullptr;
    if ((gFailFrom >= 0 && n >= gFailFrom) || bytes > gCap || gLiveBytes > gCap - bytes)
        return record(cudaErrorMemoryAllocation);
    *out = std::calloc(1, bytes ? bytes : 1);
    gLive[*out] = bytes;
    gLiveBytes += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    const auto it = gLive.find(p);
    if (it == gLive.end()) return p ? record(cudaErrorInvalidValue) : cudaSuccess;
    gBusy.clear();  // it waits for the device
    gLiveBytes -= it->second;
    std::free(p);
    gLive.erase(it);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** out, size_t bytes, unsigned) { return (*out = std::calloc(1, bytes)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t stream) {
    gBusy.insert(stream);
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t stream) {
    gBusy.insert(stream);
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = static_cast<cudaStream_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    gBusy.erase(s);
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    gBusy.erase(s);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = static_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    gBusy.clear();
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.0f;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount       ? 152
         : a == cudaDevAttrComputeCapabilityMajor  ? 10
         : a == cudaDevAttrComputeCapabilityMinor  ? 3
         : a == cudaDevAttrWarpSize                ? 32
         : a == cudaDevAttrMaxGridDimX             ? 0x7fffffff
         : a == cudaDevAttrMaxSharedMemoryPerBlock ? 49152
                                                   : 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 103;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char records[256];
    *p = records;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) { return cudaErrorInvalidValue; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = gLast;
    gLast = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return gLast; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }

}  // extern "C"
