// A stand-in for the CUDA runtime, preloaded into a child process of the tests: device memory is host memory with a limit,
// kernels do nothing, and what the host code asked for is counted. It shows how the host code behaves when the device is
// full, and what it waits for, on a machine without a GPU. Errors behave as in the runtime: a failed call stays the last
// error until someone asks cudaGetLastError.
#include <cuda_runtime_api.h>
#include <sys/mman.h>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

namespace {
std::mutex mu;
std::map<void *, size_t> live;
size_t limit = (size_t) 180 << 30, total = (size_t) 180 << 30, used = 0, largest_refused = 0;
bool refuse_pinned = false;
long long launches = 0, device_waits = 0, stream_waits = 0;
cudaStream_t last_waited = nullptr;
thread_local cudaError_t last = cudaSuccess;

cudaError_t fail(cudaError_t e) { last = e; return e; }
// (never touched until someone writes to it: a block may be larger than the machine)
void *reserve(size_t bytes) {
    void *p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    return p == MAP_FAILED ? nullptr : p;
}
int no_op() { return 0; }
}  // namespace

extern "C" {
// ---- what the tests set and read ---------------------------------------------------------------------
void fake_set_free(size_t bytes) { limit = used + bytes; }
void fake_refuse_pinned(int on) { refuse_pinned = on != 0; }
size_t fake_used() { return used; }
size_t fake_largest_refused() { return largest_refused; }
void fake_reset_counts() { launches = device_waits = stream_waits = 0; largest_refused = 0; last_waited = nullptr; }
long long fake_launches() { return launches; }
long long fake_device_waits() { return device_waits; }
long long fake_stream_waits() { return stream_waits; }

// ---- memory ------------------------------------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t bytes) {
    std::lock_guard<std::mutex> lk(mu);
    if (used + bytes > limit) {
        if (bytes > largest_refused) largest_refused = bytes;
        return fail(cudaErrorMemoryAllocation);
    }
    *p = reserve(bytes);
    if (!*p) return fail(cudaErrorMemoryAllocation);
    live[*p] = bytes;
    used += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> lk(mu);
    auto it = live.find(p);
    if (it == live.end()) return p ? fail(cudaErrorInvalidValue) : cudaSuccess;
    munmap(p, it->second);
    used -= it->second;
    live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) {
    if (refuse_pinned) return fail(cudaErrorMemoryAllocation);
    *p = calloc(1, bytes);
    return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *free_b, size_t *total_b) {
    *free_b = limit - used;
    *total_b = total;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t r = 0; r < h; ++r) memcpy((char *) d + r * dp, (const char *) s + r * sp, w);
    return cudaSuccess;
}
// (blocks of the size of a row cache are left alone)
cudaError_t cudaMemset(void *d, int v, size_t n) { if (n <= ((size_t) 64 << 20)) memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    static void *block = reserve(1 << 20);
    *p = block;
    return cudaSuccess;
}

// ---- errors, devices, kernels ------------------------------------------------------------------------
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) { *n = 74; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **p, unsigned long long, cudaDriverEntryPointQueryResult *r) {
    *p = (void *) no_op;
    if (r) *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { ++launches; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) { ++launches; return cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { ++launches; return cudaSuccess; }

// ---- streams and events ------------------------------------------------------------------------------
static cudaError_t new_stream(cudaStream_t *s) { *s = (cudaStream_t) malloc(16); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return new_stream(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return new_stream(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { ++stream_waits; last_waited = s; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { ++device_waits; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
static cudaError_t new_event(cudaEvent_t *e) { *e = (cudaEvent_t) malloc(16); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return new_event(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return new_event(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
}
