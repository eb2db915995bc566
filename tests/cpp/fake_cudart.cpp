// A stand-in for the CUDA runtime on a machine without a GPU, for tests of the
// engine's host path: device memory is host memory, kernels do not run, and
// work is complete as soon as it is enqueued. It counts what the tests ask
// about (fake_cudart.h) and fails the calls that a test tells it to fail.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>

namespace fake {
std::mutex lock;
std::map<char*, size_t> live;  // device and pinned allocations
long fail_at = -1;             // which allocation from now on fails (0: the next)
long failed = 0;
long device_syncs = 0;
long launches = 0;
bool capture_spoiled = false;
cudaStream_t capturing = nullptr;
std::thread::id capturer;

cudaError_t allocate(void** p, size_t bytes) {
    std::lock_guard<std::mutex> g(lock);
    *p = nullptr;
    if (fail_at >= 0 && fail_at-- == 0) {
        ++failed;
        return cudaErrorMemoryAllocation;
    }
    char* q = static_cast<char*>(std::calloc(1, bytes ? bytes : 1));
    live[q] = bytes;
    *p = q;
    return cudaSuccess;
}

cudaError_t release(void* p) {
    std::lock_guard<std::mutex> g(lock);
    if (!p) return cudaSuccess;
    if (!live.erase(static_cast<char*>(p))) return cudaErrorInvalidValue;
    std::free(p);
    return cudaSuccess;
}

// [p, p + bytes) lies in one live allocation, or (host memory of the caller) in none at all
bool sound(const void* p, size_t bytes) {
    std::lock_guard<std::mutex> g(lock);
    if (!p) return false;
    const char* q = static_cast<const char*>(p);
    auto it = live.upper_bound(const_cast<char*>(q));
    if (it == live.begin()) return true;
    --it;
    return q >= it->first + it->second || q + bytes <= it->first + it->second;
}

std::multiset<size_t> sizes() {
    std::lock_guard<std::mutex> g(lock);
    std::multiset<size_t> s;
    for (auto& a : live) s.insert(a.second);
    return s;
}
}  // namespace fake

namespace {
cudaError_t copy(void* dst, const void* src, size_t bytes) {
    if (bytes == 0) return cudaSuccess;
    if (!fake::sound(dst, bytes) || !fake::sound(src, bytes)) return cudaErrorInvalidValue;
    std::memmove(dst, src, bytes);
    return cudaSuccess;
}
cudaError_t fill(void* p, int v, size_t bytes) {
    if (bytes == 0) return cudaSuccess;
    if (!fake::sound(p, bytes)) return cudaErrorInvalidValue;
    std::memset(p, v, bytes);
    return cudaSuccess;
}
template <typename T>
T handle() {
    return reinterpret_cast<T>(std::malloc(1));
}
}  // namespace

extern "C" {

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "error of the stand-in"; }
cudaError_t cudaMalloc(void** p, size_t bytes) { return fake::allocate(p, bytes); }
cudaError_t cudaMallocHost(void** p, size_t bytes) { return fake::allocate(p, bytes); }
cudaError_t cudaFree(void* p) { return fake::release(p); }
cudaError_t cudaFreeHost(void* p) { return fake::release(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { return copy(d, s, n); }
cudaError_t cudaMemset(void* p, int v, size_t n) { return fill(p, v, n); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return fill(p, v, n); }

// A device must not be synchronised while one of its streams is being
// captured, by whichever thread: the call fails and the capture is lost.
cudaError_t cudaDeviceSynchronize() {
    std::lock_guard<std::mutex> g(fake::lock);
    ++fake::device_syncs;
    if (!fake::capturing) return cudaSuccess;
    fake::capture_spoiled = true;
    return cudaErrorStreamCaptureUnsupported;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    std::lock_guard<std::mutex> g(fake::lock);
    fake::capturing = s;
    fake::capturer = std::this_thread::get_id();
    fake::capture_spoiled = false;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* graph) {
    std::lock_guard<std::mutex> g(fake::lock);
    fake::capturing = nullptr;
    *graph = fake::capture_spoiled ? nullptr : handle<cudaGraph_t>();
    return fake::capture_spoiled ? cudaErrorStreamCaptureInvalidated : cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = s == fake::capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = handle<cudaStream_t>(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    return *x = handle<cudaGraphExec_t>(), cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return std::free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return std::free(x), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    return *n = 2, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, cudaErrorInvalidSymbol; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return ++fake::launches, cudaSuccess; }

// what the compiler's stubs of <<<>>> launches and its registration code call
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void*) { return *k = nullptr, cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) {
    return ++fake::launches, cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
    static void* none = nullptr;
    return &none;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"
