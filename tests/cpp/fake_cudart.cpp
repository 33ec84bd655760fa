// fake_cudart.cpp -- stands in for the CUDA runtime by LD_PRELOAD (tests/fake_runtime.py), so that the host side of
// a solve runs without a GPU: device memory is the host's, kernels do nothing, and every launch and every limit on
// a kernel's dynamic shared memory is written down. A launch above its kernel's limit fails, as does a limit above
// the device's, and other calls can be made to fail (fake_refuse).
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
struct Call {
    dim3   grid, block;
    size_t smem;
    void*  stream;
};
// less static shared memory: the most that one of the kernels holds, and that of the kernel with the highest limit
constexpr size_t kSmemDefault = 48 * 1024 - 800, kSmemOptin = 227 * 1024 - 48;
std::map<const void*, std::string> g_names;  // host stub -> kernel
std::map<const void*, size_t>      g_limits;
std::string g_log, g_refuse;
cudaError_t g_last = cudaSuccess;
Call        g_call;

const std::string& name_of(const void* f) { return g_names[f]; }
// "<call> <part of the kernel's name>"
bool refused(const char* call, const void* f) {
    const size_t sp = g_refuse.find(' ');
    return sp != std::string::npos && g_refuse.compare(0, sp, call) == 0 &&
           name_of(f).find(g_refuse.substr(sp + 1)) != std::string::npos;
}
cudaError_t fail(cudaError_t e) { return g_last = e; }
cudaError_t launched(const void* f, dim3 g, dim3 b, size_t smem) {
    if (refused("launch", f) || smem > std::max(kSmemDefault, g_limits[f])) return fail(cudaErrorInvalidValue);
    g_log += "launch " + name_of(f) + " " + std::to_string(g.x) + " " + std::to_string(b.x * b.y) + " " + std::to_string(smem) + "\n";
    return cudaSuccess;
}
}  // namespace

extern "C" {
const char* fake_kernels() {  // of every library, a line each
    static std::string all;
    all.clear();
    for (const auto& k : g_names) all += k.second + "\n";
    return all.c_str();
}
const char* fake_log() { return g_log.c_str(); }
void        fake_clear() { g_log.clear(); }
void        fake_refuse(const char* what) { g_refuse = what; }

void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { g_names[f] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
    g_call = Call{g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = g_call.grid, *b = g_call.block, *smem = g_call.smem, *(void**)s = g_call.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) { return launched((const void*)k, g, b, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return launched(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (refused("cudaFuncSetAttribute", f)) return fail(cudaErrorInvalidValue);
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    if ((size_t)v > kSmemOptin) return fail(cudaErrorInvalidValue);
    g_limits[f] = v;
    g_log += "smem " + name_of(f) + " " + std::to_string(v) + "\n";
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t, unsigned) {
    *n = refused("occupancy", f) ? 0 : 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t*) {
    *n = refused("occupancy", f) ? 0 : 16;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last              = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t) { return "refused by the test"; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::malloc(n)) ? cudaSuccess : fail(cudaErrorMemoryAllocation); }
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaFree(s); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaFree(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
}
