// Stand-in for the CUDA runtime with host memory as device memory: see alloc_main.cpp.
#include "alloc_runtime.hpp"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include <cuda_runtime_api.h>

namespace fake {
int allocs = 0, fail_at = 0, bad = 0;
std::string where;
static std::map<const char*, size_t> g_blocks;

void complain(const char* what) {
    if (++bad <= 20) std::printf("%s: %s\n", where.c_str(), what);
}
size_t blocks() { return g_blocks.size(); }
bool live(const void* p, int64_t bytes, const char* what) {
    auto it = g_blocks.upper_bound((const char*)p);
    const bool ok = p && it != g_blocks.begin() && (--it, (const char*)p + bytes <= it->first + it->second);
    if (!ok) complain(what);
    return ok;
}
Device::Device(const void* q, size_t bytes) : p(q) { g_blocks[(const char*)q] = bytes; }
Device::~Device() { g_blocks.erase((const char*)p); }
static cudaError_t take(void** p, size_t bytes) {
    *p = nullptr;
    if (++allocs == fail_at) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, bytes ? bytes : 1);
    g_blocks[(const char*)*p] = bytes;
    return cudaSuccess;
}
static cudaError_t give(void* p) {
    if (p && !g_blocks.erase((const char*)p)) complain("free of what is not allocated");
    std::free(p);
    return cudaSuccess;
}
}  // namespace fake

using namespace fake;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return take(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    if (n == 0) return cudaSuccess;
    if (k != cudaMemcpyDeviceToHost && !live(d, (int64_t)n, "copy to")) return cudaErrorInvalidValue;
    if (k != cudaMemcpyHostToDevice && !live(s, (int64_t)n, "copy from")) return cudaErrorInvalidValue;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    if (!live(d, (int64_t)n, "memset")) return cudaErrorInvalidValue;
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    *a = {};
    return cudaSuccess;  // host memory that is not pinned
}
static char g_handle;
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)&g_handle; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)&g_handle; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
}
