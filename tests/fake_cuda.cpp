// fake_cuda.cpp -- the part of the CUDA runtime that the library calls, on host memory and without
// kernels: launches do nothing and the copies are memcpy's.  Linked with the library's object
// files, it lets a CPU test make a launch, an allocation or a copy fail (fake_*), which must not be
// done to a GPU, and look at what the library does then.
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>

#include <cuda_runtime.h>

namespace {
std::mutex mu;
std::map<void*, size_t> live;
long long bytes = 0, launches = 0, allocs = 0, streams = 0;
long long fail_launch = -1, fail_alloc = -1;    // the launch or allocation (counted from 0) that fails
const void* fail_copy = nullptr;                // a copy to this address fails
std::map<const void*, int> smem;                // a kernel's opt-in
long long lowered = 0;
long long answer_at = -1;                       // the 4-byte copy that brings `answer`
long long copies4 = 0;
int answer = 0;
void* word = nullptr;                           // the first 4-byte memset since fake_reset
cudaError_t last = cudaSuccess;
int slow_stream_ms = 0;

void* take(size_t n)
{
    void* p = std::calloc(1, n ? n : 1);
    std::lock_guard<std::mutex> lk(mu);
    live[p] = n;
    bytes += (long long)n;
    return p;
}
cudaError_t launch()
{
    std::lock_guard<std::mutex> lk(mu);
    if (launches++ == fail_launch) return last = cudaErrorLaunchOutOfResources;
    return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- what the tests call
void fake_reset()
{
    std::lock_guard<std::mutex> lk(mu);
    launches = allocs = 0;
    fail_launch = fail_alloc = -1;
    fail_copy = nullptr;
    word = nullptr;
    answer_at = -1;
    copies4 = 0;
    last = cudaSuccess;
}
void fake_fail_launch(long long k) { fail_launch = k; }
void fake_fail_allocs_from(long long k) { fail_alloc = k; }
void fake_fail_copy_to(const void* p) { fail_copy = p; }
void fake_answer(long long k, int v) { answer_at = k; answer = v; }
void fake_slow_streams(int ms) { slow_stream_ms = ms; }
long long fake_launches() { return launches; }
long long fake_allocs() { return allocs; }
long long fake_bytes() { return bytes; }
long long fake_streams() { return streams; }
long long fake_lowered() { return lowered; }
int* fake_word() { return static_cast<int*>(word); }

// ---- memory
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t)
{
    {
        std::lock_guard<std::mutex> lk(mu);
        if (fail_alloc >= 0 && allocs >= fail_alloc) return last = cudaErrorMemoryAllocation;
        ++allocs;
    }
    *p = take(n);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t)
{
    std::lock_guard<std::mutex> lk(mu);
    auto it = live.find(p);
    if (it == live.end()) return last = cudaErrorInvalidValue;
    bytes -= (long long)it->second;
    live.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (d == fail_copy) return last = cudaErrorUnknown;
    std::memcpy(d, s, n);
    if (n == 4 && copies4++ == answer_at) *static_cast<int*>(d) = answer;
    if (n == 12) *static_cast<int*>(d) = 1;     // (an expansion's flags: done)
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t)
{
    if (n == 4 && !word) word = p;
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 33; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = reinterpret_cast<cudaMemPool_t>(&live); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { std::memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaErrorInvalidSymbol; }

// ---- device, streams, events
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof(*p)); p->totalGlobalMem = (size_t)1 << 33; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaGetLastError()
{
    std::lock_guard<std::mutex> lk(mu);
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    std::this_thread::sleep_for(std::chrono::milliseconds(slow_stream_ms));
    std::lock_guard<std::mutex> lk(mu);
    *s = reinterpret_cast<cudaStream_t>(++streams << 4);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = static_cast<cudaEvent_t>(take(8)); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaFreeAsync(e, nullptr); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

// ---- kernels
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v)
{
    std::lock_guard<std::mutex> lk(mu);
    int& have = smem[f];
    if (v < have) ++lowered;
    have = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return launch(); }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f)); return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st)
{
    *g = *b = dim3(1);
    *s = 0;
    *static_cast<void**>(st) = nullptr;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"
