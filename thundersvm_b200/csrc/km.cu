// KernelMatrix on the device: construction, self dots / diagonal, and kernel rows for the
// CSR engine and the CUDA-core dense engine. The tensor-core dense engine lives in
// dense_tc.cu. Reference behaviour: src/thundersvm/kernelmatrix.cpp:183-316,385-406.
#include "common.cuh"
#include <cuda_fp16.h>
#include <string.h>
#include <stdlib.h>
#include <atomic>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace tsvm {

static thread_local char g_err[512] = "";
static std::atomic<long long> g_launches{0};

void set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
long long launch_count() { return g_launches.load(); }
void count_launch(int k) { g_launches.fetch_add(k); }

// ---- memory pool -------------------------------------------------------------------------------------
// Size classes: eight per power of two (at most 12.5 % slack), 512 bytes at least. Blocks are per device.
namespace {
struct PoolBlock { int dev; size_t cls; };
// never destroyed: handles may be released after the static destructors of this library have run
std::mutex &g_pool_mu = *new std::mutex;
auto &g_pool_live = *new std::unordered_map<void *, PoolBlock>;
auto &g_pinned_live = *new std::unordered_map<void *, PoolBlock>;
auto &g_pool_free = *new std::map<std::pair<int, size_t>, std::vector<void *>>;
auto &g_pinned_free = *new std::map<size_t, std::vector<void *>>;
size_t g_pool_cached = 0;               // bytes in g_pool_free
size_t g_pinned_cached = 0;             // bytes in g_pinned_free
constexpr size_t MAX_PINNED_CACHED = 64 << 20;

size_t size_class(size_t bytes) {
    if (bytes < 512) return 512;
    size_t p2 = 512;
    while (p2 < bytes) p2 <<= 1;          // smallest power of two >= bytes
    const size_t step = p2 >> 4;          // eighths of the previous power of two
    return (bytes + step - 1) / step * step;
}
}  // namespace

void pool_release() {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    int cur = 0;
    cudaGetDevice(&cur);
    for (auto &kv : g_pool_free) {
        if (kv.second.empty()) continue;
        cudaSetDevice(kv.first.first);
        for (void *q : kv.second) cudaFree(q);
        kv.second.clear();
    }
    g_pool_cached = 0;
    cudaSetDevice(cur);
    for (auto &kv : g_pinned_free) {
        for (void *q : kv.second) cudaFreeHost(q);
        kv.second.clear();
    }
    g_pinned_cached = 0;
}

tsvm_status pool_alloc(void **p, size_t bytes) {
    *p = nullptr;
    int dev = 0;
    TSVM_CUDA(cudaGetDevice(&dev));
    const size_t cls = size_class(bytes);
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        auto it = g_pool_free.find({dev, cls});
        if (it != g_pool_free.end() && !it->second.empty()) {
            *p = it->second.back();
            it->second.pop_back();
            g_pool_cached -= cls;
            g_pool_live[*p] = PoolBlock{dev, cls};
            return TSVM_OK;
        }
    }
    cudaError_t e = cudaMalloc(p, cls);
    if (e == cudaErrorMemoryAllocation) {      // give the cached blocks back and try once more
        cudaGetLastError();
        pool_release();
        e = cudaMalloc(p, cls);
    }
    TSVM_CUDA(e);
    std::lock_guard<std::mutex> lk(g_pool_mu);
    g_pool_live[*p] = PoolBlock{dev, cls};
    return TSVM_OK;
}

// A freed block may be handed out again at once, so nothing in flight may still use it: one wait per device
// that owns one of the blocks (the owning device, which need not be the caller's current one), then all of
// them go to the free lists. Cached bytes above the cap go back to the driver, largest blocks first.
static size_t pool_cache_cap() {
    // TSVM_POOL_CACHE_MB, else 60 % of the current device's memory (a solver's row cache is the largest block and
    // should come back from the pool when the next solver of the same problem is created)
    static const size_t cap = [] {
        if (const char *e = getenv("TSVM_POOL_CACHE_MB")) return (size_t) strtoull(e, nullptr, 10) << 20;
        return (size_t) ((double) device_memory_bytes() * 0.6);
    }();
    return cap;
}

// cudaMemGetInfo takes a driver lock that other processes of the machine hold too: usually 100 us, at times 40 ms. What
// the library wants to know is the size of the device, which does not change.
int device_sm_count() {
    static std::atomic<int> count[MAX_DEVICES];
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return sms; }
    std::atomic<int> &known = count[dev & (MAX_DEVICES - 1)];
    if (const int k = known.load(std::memory_order_relaxed)) return k;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) cudaGetLastError();
    known.store(sms, std::memory_order_relaxed);
    return sms;
}

size_t device_l2_bytes() {
    static std::atomic<int> bytes[MAX_DEVICES];
    int dev = 0, size = 126 << 20;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return size; }
    std::atomic<int> &known = bytes[dev & (MAX_DEVICES - 1)];
    if (const int k = known.load(std::memory_order_relaxed)) return k;
    if (cudaDeviceGetAttribute(&size, cudaDevAttrL2CacheSize, dev) != cudaSuccess) cudaGetLastError();
    known.store(size, std::memory_order_relaxed);
    return size;
}

size_t device_memory_bytes() {
    static std::atomic<size_t> bytes[MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return (size_t) 32 << 30; }
    std::atomic<size_t> &known = bytes[dev & (MAX_DEVICES - 1)];
    size_t total = known.load(std::memory_order_relaxed);
    if (total) return total;
    size_t free_b = 0;
    if (cudaMemGetInfo(&free_b, &total) != cudaSuccess) { cudaGetLastError(); return (size_t) 32 << 30; }
    known.store(total, std::memory_order_relaxed);
    return total;
}

void pool_free_many(std::initializer_list<void *> blocks, bool idle) {
    int cur = 0;
    bool have_cur = false;
    unsigned long long synced = 0;
    std::vector<void *> foreign;
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        for (void *p : blocks) {
            if (!p) continue;
            auto it = g_pool_live.find(p);
            if (it == g_pool_live.end()) { foreign.push_back(p); continue; }
            if (!idle) synced |= 1ull << (it->second.dev & (MAX_DEVICES - 1));
        }
    }
    for (int dev = 0; dev < MAX_DEVICES; ++dev) {
        if (!((synced >> dev) & 1ull)) continue;
        if (!have_cur) { cudaGetDevice(&cur); have_cur = true; }
        if (dev != cur) cudaSetDevice(dev);
        cudaDeviceSynchronize();
        if (dev != cur) cudaSetDevice(cur);
    }
    for (void *p : foreign) cudaFree(p);                     // not ours (never happens for handle memory)
    std::vector<std::pair<int, void *>> to_driver;
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        for (void *p : blocks) {
            if (!p) continue;
            auto it = g_pool_live.find(p);
            if (it == g_pool_live.end()) continue;
            g_pool_free[{it->second.dev, it->second.cls}].push_back(p);
            g_pool_cached += it->second.cls;
            g_pool_live.erase(it);
        }
        // over the cap: return the largest cached blocks first
        for (auto kv = g_pool_free.rbegin(); kv != g_pool_free.rend() && g_pool_cached > pool_cache_cap(); ++kv)
            while (!kv->second.empty() && g_pool_cached > pool_cache_cap()) {
                to_driver.push_back({kv->first.first, kv->second.back()});
                kv->second.pop_back();
                g_pool_cached -= kv->first.second;
            }
    }
    for (auto &b : to_driver) {
        if (!have_cur) { cudaGetDevice(&cur); have_cur = true; }
        if (b.first != cur) cudaSetDevice(b.first);
        cudaFree(b.second);
        if (b.first != cur) cudaSetDevice(cur);
    }
}

void pool_free(void *p) {
    if (p) pool_free_many({p});
}

tsvm_status pinned_alloc(void **p, size_t bytes) {
    *p = nullptr;
    const size_t cls = size_class(bytes);
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        auto &v = g_pinned_free[cls];
        if (!v.empty()) {
            *p = v.back();
            v.pop_back();
            g_pinned_cached -= cls;
            g_pinned_live[*p] = PoolBlock{0, cls};
            return TSVM_OK;
        }
    }
    TSVM_CUDA(cudaMallocHost(p, cls));
    std::lock_guard<std::mutex> lk(g_pool_mu);
    g_pinned_live[*p] = PoolBlock{0, cls};
    return TSVM_OK;
}

void pinned_free(void *p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pinned_live.find(p);
    if (it == g_pinned_live.end()) { cudaFreeHost(p); return; }
    if (g_pinned_cached + it->second.cls > MAX_PINNED_CACHED) cudaFreeHost(p);
    else {
        g_pinned_free[it->second.cls].push_back(p);
        g_pinned_cached += it->second.cls;
    }
    g_pinned_live.erase(it);
}

tsvm_status launch_dense_tc(tsvm_km *km, int m, float *out, long long ld_out, cudaStream_t st);  // dense_tc.cu

// ---- construction kernels ---------------------------------------------------------------

// diag (kernelmatrix.cpp:225-247)
__device__ __forceinline__ float diag_value(const KernelFn &fn, float v) {
    switch (fn.type) {
        case TSVM_RBF: case TSVM_PRECOMPUTED: return 1.0f;
        case TSVM_POLY: return powf(fn.gamma * v + fn.coef0, (float) fn.degree);
        case TSVM_SIGMOID: return tanhf(fn.gamma * v + fn.coef0);
        default: return v;
    }
}

// Self dots float(sum_k double(x_ik)^2) and diagonal of CSR instances, one warp per row (kernelmatrix.cpp:194-247).
__global__ void self_dot_csr_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr, int n, KernelFn fn,
                                    float *__restrict__ sd, float *__restrict__ diag, int *__restrict__ status) {
    int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x < 4) status[threadIdx.x] = 0;
    if (row >= n) return;
    double s = 0;
    for (int p = row_ptr[row] + lane; p < row_ptr[row + 1]; p += 32) { double v = val[p]; s += v * v; }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) { sd[row] = (float) s; diag[row] = diag_value(fn, (float) s); }
}

// Self dots of a batch of new instances, accumulated sequentially in float in storage order as kernelmatrix.cpp:288-296
// does: one thread per row keeps that order. What bounds it is that chain, 4 cycles per feature; the rows have to be
// there in time. A warp copies 32 rows x 64 features at a time (asynchronous copies, coalesced, four stages in flight) to
// shared memory and each lane adds up its own row from there: 4,096 rows x 2,000 155 -> 23 us against loads that every lane
// made from its own row. VEC: 16-byte copies (aligned rows), else 4-byte ones.
constexpr int SEQ_COLS = 64, SEQ_STAGES = 4, SEQ_LD = SEQ_COLS + 4;      // row stride: 16-byte reads without bank conflicts
template <bool VEC>
__device__ __forceinline__ void self_dots_of_32_rows(const float *__restrict__ T, int r0, int m, int dt, int ldt,
                                                     float (*tile)[32][SEQ_LD], float *__restrict__ out) {
    const int lane = threadIdx.x & 31, blocks = (dt + SEQ_COLS - 1) / SEQ_COLS;
    auto fetch = [&](int kb) {
        if (kb < blocks) {
            constexpr int W = VEC ? 4 : 1, PER_ROW = SEQ_COLS / W;
#pragma unroll 8
            for (int e = lane; e < 32 * PER_ROW; e += 32) {
                const int r = e / PER_ROW, c = (e % PER_ROW) * W, k = kb * SEQ_COLS + c;
                int bytes = (dt - k) * 4;                               // beyond the row's end: zeros, which add nothing
                bytes = r0 + r < m && bytes > 0 ? (bytes < W * 4 ? bytes : W * 4) : 0;
                const float *src = bytes ? T + (size_t) (r0 + r) * ldt + k : T;
                const unsigned dst = (unsigned) __cvta_generic_to_shared(&tile[kb % SEQ_STAGES][r][c]);
                if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
                else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int kb = 0; kb < SEQ_STAGES - 1; ++kb) fetch(kb);
    float s = 0;
    for (int kb = 0; kb < blocks; ++kb) {
        fetch(kb + SEQ_STAGES - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(SEQ_STAGES - 1) : "memory");
        __syncwarp();
        const float *x = tile[kb % SEQ_STAGES][lane];
#pragma unroll
        for (int c = 0; c < SEQ_COLS; c += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(x + c);
            s = fmaf(v.x, v.x, s); s = fmaf(v.y, v.y, s); s = fmaf(v.z, v.z, s); s = fmaf(v.w, v.w, s);
        }
        __syncwarp();
    }
    if (r0 + lane < m) out[r0 + lane] = s;
}

template <bool VEC>
__global__ void __launch_bounds__(32) self_dot_seq_dense_kernel(const float *__restrict__ T, int m, int dt, int ldt,
                                                                float *__restrict__ out) {
    __shared__ __align__(16) float tile[SEQ_STAGES][32][SEQ_LD];
    self_dots_of_32_rows<VEC>(T, blockIdx.x * 32, m, dt, ldt, tile, out);
}

static tsvm_status launch_self_dot_seq_dense(const float *T, int m, int dt, int ldt, float *out, cudaStream_t st) {
    if ((ldt & 3) == 0 && ((uintptr_t) T & 15) == 0)
        TSVM_LAUNCH(self_dot_seq_dense_kernel<true>, ceil_div(m, 32), 32, 0, st, T, m, dt, ldt, out);
    else TSVM_LAUNCH(self_dot_seq_dense_kernel<false>, ceil_div(m, 32), 32, 0, st, T, m, dt, ldt, out);
    return TSVM_OK;
}

__device__ __forceinline__ float self_dot_seq_csr(const float *__restrict__ val, int begin, int end) {
    float s = 0;
    for (int p = begin; p < end; ++p) s = fmaf(val[p], val[p], s);
    return s;
}
__global__ void self_dot_seq_csr_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr, int m,
                                        float *__restrict__ out) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < m) out[r] = self_dot_seq_csr(val, row_ptr[r], row_ptr[r + 1]);
}

// TF32 split x = hi + lo (+ <= 2^-22 |x|): hi = x rounded to TF32, lo = (x - hi) rounded to
// TF32, both with the 13 low mantissa bits cleared so that the tensor core reads exactly
// these values whether it truncates or rounds its FP32 operands.
__device__ __forceinline__ void split_tf32(float x, float &hi, float &lo) {
    unsigned h, l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
    hi = __uint_as_float(h);
    float r = x - hi;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(r));
    lo = __uint_as_float(l);
}

// Row-scaled FP16 split: the row is multiplied by a power of two that puts its largest magnitude in
// [2^14, 2^15), then x*scale = hi + lo (+ <= 2^-24 |x*scale|) with hi, lo FP16 (lo may be subnormal:
// absolute precision 2^-24, i.e. 2^-39 of the row maximum). Products of FP16 values are exact in the
// tensor core's FP32 accumulator, and the epilogue multiplies the sum by the two rows' 1/scale.
__device__ __forceinline__ void row_scale_from_max(float amax, float &scale, float &unscale) {
    const int ex = (int) ((__float_as_uint(amax) >> 23) & 0xffu) - 127;
    int se = (ex == -127) ? 0 : 14 - ex;          // all-zero (or denormal) rows stay unscaled
    se = se < -126 ? -126 : (se > 126 ? 126 : se);
    scale = __uint_as_float((unsigned) (se + 127) << 23);
    unscale = __uint_as_float((unsigned) (127 - se) << 23);
}

__device__ __forceinline__ void split_f16(float xs, __half &hi, __half &lo) {
    hi = __float2half_rn(xs);
    lo = __float2half_rn(xs - __half2float(hi));
}

// plane_kind 1: TF32 words; 2: FP16 halves of the scaled value (off counts elements of the plane).
__device__ __forceinline__ void store_planes(int kind, float *hi, float *lo, size_t off, float v, float scale) {
    if (kind == 2) {
        __half h, l;
        split_f16(v * scale, h, l);
        reinterpret_cast<__half *>(hi)[off] = h;
        reinterpret_cast<__half *>(lo)[off] = l;
    } else {
        float h, l;
        split_tf32(v, h, l);
        hi[off] = h;
        lo[off] = l;
    }
}

// max |v| over the block (every thread calls it once per kernel; blockDim a multiple of 32, <= 1024)
__device__ __forceinline__ float block_max_abs(float v) {
    __shared__ unsigned red[32];
    const unsigned full = 0xffffffffu;
    unsigned b = __reduce_max_sync(full, __float_as_uint(fabsf(v)));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = b;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    b = (int) (threadIdx.x & 31) < nw ? red[threadIdx.x & 31] : 0u;
    return __uint_as_float(__reduce_max_sync(full, b));
}

// Where the staging kernels put a requested row: FP32 W (CUDA-core engine) or the two planes.
struct RowDst {
    float *W, *hi, *lo, *unscale;
    int kind, ld;                  // plane kind (0 = FP32 W) and row length in elements
};

// Self dots, diagonal and operand planes of all instances: one warp per row, one pass over X (the second look at a row
// comes from L1). kind 0: no planes. sd == nullptr: planes only. Columns d..pld-1 of the planes are zero.
__global__ void prepare_rows_kernel(const float *__restrict__ X, int n, int d, int ld, int kind, int pld,
                                    float *__restrict__ hi, float *__restrict__ lo, float *__restrict__ x_unscale, KernelFn fn,
                                    float *__restrict__ sd, float *__restrict__ diag, int *__restrict__ status) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    if (sd && blockIdx.x == 0 && threadIdx.x < 4) status[threadIdx.x] = 0;
    for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < n; row += gridDim.x * wpb) {
        const float *x = X + (size_t) row * ld;
        float amax = 0.0f;
        double s = 0;
#pragma unroll 4
        for (int k = lane; k < d; k += 32) {
            const float v = x[k];
            amax = fmaxf(amax, fabsf(v));
            s += (double) v * v;
        }
        if (sd) {
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) { sd[row] = (float) s; diag[row] = diag_value(fn, (float) s); }
        }
        if (kind == 0) continue;
        float scale = 1.0f, unscale = 1.0f;
        if (kind == 2) {
            amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
            row_scale_from_max(amax, scale, unscale);
            if (lane == 0) x_unscale[row] = unscale;
        }
#pragma unroll 4
        for (int k = lane; k < pld; k += 32)
            store_planes(kind, hi, lo, (size_t) row * pld + k, k < d ? x[k] : 0.0f, scale);
    }
}

// ---- gathering the requested rows ----------------------------------------------------------

// Requested row i = X[idx[i]][0..d) (zero padded to the destination's row length); sd_rows[i].
__global__ void gather_rows_dense_kernel(const float *__restrict__ X, int ld, int d, const int *__restrict__ idx,
                                         int m, const float *__restrict__ sd, RowDst dst,
                                         float *__restrict__ sd_rows, const int *__restrict__ m_dev) {
    int i = blockIdx.x;
    if (i >= m || (m_dev && i >= *m_dev)) return;
    const int r = idx[i];
    const int dr = r >= 0 ? d : 0;           // id -1 (an empty working-set slot) is staged as an all-zero row
    const float *x = X + (size_t) (r >= 0 ? r : 0) * ld;
    float scale = 1.0f, unscale = 1.0f;
    if (dst.kind == 2) {
        float amax = 0.0f;
        for (int k = threadIdx.x; k < dr; k += blockDim.x) amax = fmaxf(amax, fabsf(x[k]));
        row_scale_from_max(block_max_abs(amax), scale, unscale);
        if (threadIdx.x == 0) dst.unscale[i] = unscale;
    }
    for (int k = threadIdx.x; k < dst.ld; k += blockDim.x) {
        float v = k < dr ? x[k] : 0.0f;
        if (dst.W) dst.W[(size_t) i * dst.ld + k] = v;
        else store_planes(dst.kind, dst.hi, dst.lo, (size_t) i * dst.ld + k, v, scale);
    }
    if (threadIdx.x == 0) sd_rows[i] = r >= 0 ? sd[r] : 0.0f;
}

// Same for a batch of new dense instances T (m x dt, stride ldt); features >= d are dropped.
__global__ void stage_rows_dense_kernel(const float *__restrict__ T, int ldt, int dt, int d, int m, RowDst dst) {
    int i = blockIdx.x;
    if (i >= m) return;
    const float *x = T + (size_t) i * ldt;
    const int lim = d < dt ? d : dt;
    float scale = 1.0f, unscale = 1.0f;
    if (dst.kind == 2) {
        float amax = 0.0f;
        for (int k = threadIdx.x; k < lim; k += blockDim.x) amax = fmaxf(amax, fabsf(x[k]));
        row_scale_from_max(block_max_abs(amax), scale, unscale);
        if (threadIdx.x == 0) dst.unscale[i] = unscale;
    }
    for (int k = threadIdx.x; k < dst.ld; k += blockDim.x) {
        float v = k < lim ? x[k] : 0.0f;
        if (dst.W) dst.W[(size_t) i * dst.ld + k] = v;
        else store_planes(dst.kind, dst.hi, dst.lo, (size_t) i * dst.ld + k, v, scale);
    }
}

// Which storage CSR data is worked on in. With at least CSR_DENSE_SHARE of the entries present (or at most 256 features)
// the tensor-core engine needs less time for whole rows than the CSR engine for the entries: 512 rows of 32,561 instances,
// 14 of 123 features set, take 103 us with the entries and 51 us as dense rows; predicting 16,281 rows with 12,001 of
// them 1.7 and 0.53 ms. That engine splits a value into two FP16 planes, so the rule asks for data that one FP16 number
// holds exactly (one-hot and binary features, small counts): the products are exact and nothing is rounded that the CSR
// engine does not round. The features of a row also have to be strictly ascending: one that occurs twice counts twice
// in the CSR engine. Below 33 features dense rows run on CUDA cores.
constexpr double CSR_DENSE_SHARE = 0.02;
constexpr int CSR_DENSE_MIN_D = 33, CSR_DENSE_ANY_D = 256, CSR_DENSE_MAX_D = 4096;

// out[0] = 1 if some entry rules the dense form out, out[1] = row_ptr[n] (both zeroed before). batch: rows to predict,
// staged by assignment and cut at d in either form, so only their values count.
__global__ void inspect_entries_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr,
                                       const int *__restrict__ col, int n, int d, bool batch, int *__restrict__ out) {
    if (blockIdx.x == 0 && threadIdx.x == 0) out[1] = row_ptr[n];
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    bool bad = false;
    for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < n && !bad; row += gridDim.x * wpb) {
        const int b = row_ptr[row], e = row_ptr[row + 1];
        for (int p = b + lane; p < e; p += 32) {
            const float v = val[p], a = fabsf(v);
            // 2^-10 .. 2^5: inside one row's scaling every such value keeps its eleven bits
            const bool exact = v == 0.0f || (a >= 0.0009765625f && a <= 32.0f && __half2float(__float2half_rn(v)) == v);
            bad |= !exact || (!batch && (col[p] < 0 || col[p] >= d || (p > b && col[p - 1] >= col[p])));
        }
        bad = __any_sync(0xffffffffu, bad);
    }
    if (bad && lane == 0) out[0] = 1;
}

__global__ void dense_from_csr_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr,
                                      const int *__restrict__ col, int n, int ld, float *__restrict__ X) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < n; row += gridDim.x * wpb) {
        float *x = X + (size_t) row * ld;
        for (int k = lane; k < ld; k += 32) x[k] = 0.0f;
        __syncwarp();
        for (int p = row_ptr[row] + lane; p < row_ptr[row + 1]; p += 32) x[col[p]] = val[p];
    }
}

// A batch of new instances as the requested rows of a dense engine, in one launch whose blocks do different things: the
// self dots (a chain per row: the longest part, so these blocks come first), the rows in the engine's operand form (a warp
// per row; features >= d are dropped) and, for the fused prediction, -rho into the sums that the contraction adds to.
// Separate launches took the sum of their times and a launch each: 8 + 8.5 + 2 us per 4,096 rows of 784 features, most
// of it latency, against 10.9 us.
constexpr int BATCH_THREADS = 128, BATCH_WARPS = BATCH_THREADS / 32;
__device__ __forceinline__ void preset_sums(const SumPreset &p, int block) {
    const long long e = (long long) block * BATCH_THREADS + threadIdx.x;
    if (e < p.total) p.sums[e] = -p.rho[p.pair_stride == 1 ? e % p.n_pairs : e / p.pair_stride];
}

template <bool VEC>
__global__ void __launch_bounds__(BATCH_THREADS)
stage_batch_dense_kernel(const float *__restrict__ T, int ldt, int dt, int d, int m, RowDst dst, float *__restrict__ sd,
                         int dot_blocks, int row_blocks, const SumPreset preset) {
    __shared__ __align__(16) float tile[SEQ_STAGES][32][SEQ_LD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int) blockIdx.x < dot_blocks) {
        if (warp == 0) self_dots_of_32_rows<VEC>(T, blockIdx.x * 32, m, dt, ldt, tile, sd);
        return;
    }
    const int block = blockIdx.x - dot_blocks;
    if (block >= row_blocks) return preset_sums(preset, block - row_blocks);
    const int lim = d < dt ? d : dt;
    for (int i = block * BATCH_WARPS + warp; i < m; i += row_blocks * BATCH_WARPS) {
        const float *x = T + (size_t) i * ldt;
        // four features at a time (VEC: one 16-byte load)
        auto four = [&](int k, float (&v)[4]) {
            if (VEC && k + 3 < lim) {
                const float4 t = *reinterpret_cast<const float4 *>(x + k);
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = k + u < lim ? x[k + u] : 0.0f;
            }
        };
        float scale = 1.0f, unscale = 1.0f;
        if (dst.kind == 2) {
            float amax = 0.0f;
#pragma unroll 4
            for (int k = 4 * lane; k < lim; k += 128) {
                float v[4];
                four(k, v);
                amax = fmaxf(fmaxf(fmaxf(amax, fabsf(v[0])), fmaxf(fabsf(v[1]), fabsf(v[2]))), fabsf(v[3]));
            }
            amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
            row_scale_from_max(amax, scale, unscale);
            if (lane == 0) dst.unscale[i] = unscale;
        }
#pragma unroll 4
        for (int k = 4 * lane; k < dst.ld; k += 128) {          // (a row of the destination is a multiple of four long)
            float v[4];
            four(k, v);
            const size_t at = (size_t) i * dst.ld + k;
            if (dst.W) *reinterpret_cast<float4 *>(dst.W + at) = make_float4(v[0], v[1], v[2], v[3]);
            else if (dst.kind == 2) {
                __half h[4], l[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) split_f16(v[u] * scale, h[u], l[u]);
                *reinterpret_cast<uint2 *>(reinterpret_cast<__half *>(dst.hi) + at) = *reinterpret_cast<const uint2 *>(h);
                *reinterpret_cast<uint2 *>(reinterpret_cast<__half *>(dst.lo) + at) = *reinterpret_cast<const uint2 *>(l);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) store_planes(dst.kind, dst.hi, dst.lo, at + u, v[u], scale);
            }
        }
    }
}

__global__ void __launch_bounds__(BATCH_THREADS)
stage_batch_csr_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr, const int *__restrict__ col, int m, int d,
                       RowDst dst, float *__restrict__ sd, int dot_blocks, int row_blocks, const SumPreset preset) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int) blockIdx.x < dot_blocks) {
        const int r = blockIdx.x * BATCH_THREADS + threadIdx.x;
        if (r < m) sd[r] = self_dot_seq_csr(val, row_ptr[r], row_ptr[r + 1]);
        return;
    }
    const int block = blockIdx.x - dot_blocks;
    if (block >= row_blocks) return preset_sums(preset, block - row_blocks);
    for (int i = block * BATCH_WARPS + warp; i < m; i += row_blocks * BATCH_WARPS) {
        const int b = row_ptr[i], e = row_ptr[i + 1];
        float amax = 0.0f, scale = 1.0f, unscale = 1.0f;
        const size_t at = (size_t) i * dst.ld;
        if (dst.W) {
            for (int k = 4 * lane; k < dst.ld; k += 128) *reinterpret_cast<float4 *>(dst.W + at + k) = make_float4(0, 0, 0, 0);
        } else if (dst.kind == 2) {
            for (int p = b + lane; p < e; p += 32)
                if (col[p] < d) amax = fmaxf(amax, fabsf(val[p]));
            amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
            row_scale_from_max(amax, scale, unscale);
            if (lane == 0) dst.unscale[i] = unscale;
            for (int k = 8 * lane; k < dst.ld; k += 256) {      // (a multiple of eight halves)
                *reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(dst.hi) + at + k) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(dst.lo) + at + k) = make_uint4(0, 0, 0, 0);
            }
        } else {
            for (int k = 4 * lane; k < dst.ld; k += 128) {
                *reinterpret_cast<float4 *>(dst.hi + at + k) = make_float4(0, 0, 0, 0);
                *reinterpret_cast<float4 *>(dst.lo + at + k) = make_float4(0, 0, 0, 0);
            }
        }
        __syncwarp();                                           // the zeros are in place before the entries
        for (int p = b + lane; p < e; p += 32) {
            const int c = col[p];
            if (c >= d) continue;
            if (dst.W) dst.W[at + c] = val[p];
            else store_planes(dst.kind, dst.hi, dst.lo, at + c, val[p], scale);
        }
        __syncwarp();
    }
}

constexpr int CSR_PART = 128;               // requested rows per part of the CSR engine

// CSR engine staging: WT[c * wt_ld + i] = value of feature c in requested row i, and a bit for feature c in the bitmap
// of row i's part (bits [parts][words], words == 0: none). Both are kept all-zero between calls: `clear` = true writes
// zeros back at the same places.
__global__ void scatter_csr_to_wt_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr,
                                         const int *__restrict__ col, const int *__restrict__ idx, int m, int d,
                                         int wt_ld, float *__restrict__ WT, const float *__restrict__ sd,
                                         float *__restrict__ sd_rows, bool clear, const int *__restrict__ m_dev,
                                         unsigned *__restrict__ bits, int words) {
    int i = blockIdx.x;
    if (i >= m || (m_dev && i >= *m_dev)) return;
    int r = idx ? idx[i] : i;
    if (r < 0) {                             // an empty working-set slot: an all-zero row
        if (!clear && sd && threadIdx.x == 0) sd_rows[i] = 0.0f;
        return;
    }
    unsigned *mine = bits + (size_t) (i / CSR_PART) * words;
    for (int p = row_ptr[r] + threadIdx.x; p < row_ptr[r + 1]; p += blockDim.x) {
        int c = col[p];
        if (c >= d) continue;
        WT[(size_t) c * wt_ld + i] = clear ? 0.0f : val[p];
        if (words) {
            if (clear) mine[c >> 5] = 0u;
            else atomicOr(mine + (c >> 5), 1u << (c & 31));
        }
    }
    if (!clear && sd && threadIdx.x == 0) sd_rows[i] = sd[r];
}

// WT from a dense batch T (m x dt): WT[c * wt_ld + i] = T[i][c] for c < min(d, dt).
__global__ void transpose_dense_to_wt_kernel(const float *__restrict__ T, int ldt, int dt, int d, int m, int wt_ld,
                                             float *__restrict__ WT, bool clear) {
    __shared__ float tile[32][33];
    int c0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
    int tx = threadIdx.x, ty = threadIdx.y;   // 32 x 8
    int lim = d < dt ? d : dt;
    for (int r = ty; r < 32; r += 8) {
        int i = i0 + r, c = c0 + tx;
        tile[r][tx] = (!clear && i < m && c < lim) ? T[(size_t) i * ldt + c] : 0.0f;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        int c = c0 + r, i = i0 + tx;
        if (c < d && i < m) WT[(size_t) c * wt_ld + i] = tile[tx][r];
    }
}

// Operand planes, self dots and 1/scale of the instances ids[0..m) copied out of the kernel matrix's planes
// (row_bytes a multiple of 16).
__global__ void gather_planes_kernel(const float *__restrict__ Xhi, const float *__restrict__ Xlo, size_t row_bytes,
                                     const int *__restrict__ ids, int m, const float *__restrict__ sd,
                                     const float *__restrict__ x_unscale, float *__restrict__ hi,
                                     float *__restrict__ lo, float *__restrict__ sd_out,
                                     float *__restrict__ unscale_out, const int *__restrict__ m_dev) {
    const int i = blockIdx.x;
    if (i >= m || (m_dev && i >= *m_dev)) return;
    const int r = ids[i] >= 0 ? ids[i] : 0;      // an empty slot copies some row; its y = 0 keeps it inert
    const size_t vecs = row_bytes / 16;
    const uint4 *sh = reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(Xhi) + (size_t) r * row_bytes);
    const uint4 *sl = reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(Xlo) + (size_t) r * row_bytes);
    uint4 *dh = reinterpret_cast<uint4 *>(reinterpret_cast<char *>(hi) + (size_t) i * row_bytes);
    uint4 *dl = reinterpret_cast<uint4 *>(reinterpret_cast<char *>(lo) + (size_t) i * row_bytes);
    for (size_t v = threadIdx.x; v < vecs; v += blockDim.x) { dh[v] = sh[v]; dl[v] = sl[v]; }
    if (threadIdx.x == 0) { sd_out[i] = sd[r]; unscale_out[i] = x_unscale ? x_unscale[r] : 1.0f; }
}

// ---- CUDA-core dense engine: out[i][j] = kfn(sum_k W[i][k] X[j][k]) -------------------------
// 64 instances x 64 requested rows per block, 16-wide k slabs, 4x4 outputs per thread.
__global__ void __launch_bounds__(256)
dense_rows_simt_kernel(const float *__restrict__ X, int ldx, int n, const float *__restrict__ W, int ldw, int m_launch,
                       int d_pad, const float *__restrict__ sd, const float *__restrict__ sd_rows, KernelFn fn,
                       float *__restrict__ out, long long ld_out, const int *__restrict__ m_dev,
                       const int *__restrict__ row_slot) {
    __shared__ float xs[16][64 + 4];
    __shared__ float wsm[16][64 + 4];
    const int m = m_dev ? min(m_launch, max(*m_dev, 0)) : m_launch;     // the count found on the device, if any
    const int j0 = blockIdx.x * 64, i0 = blockIdx.y * 64;
    if (i0 >= m) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
    const int lr = tid >> 2, lk = (tid & 3) * 4;   // 64 rows x 4 float4 per slab
    for (int k0 = 0; k0 < d_pad; k0 += 16) {
        float4 xv = make_float4(0, 0, 0, 0), wv = make_float4(0, 0, 0, 0);
        if (j0 + lr < n && k0 + lk < d_pad) xv = *reinterpret_cast<const float4 *>(X + (size_t) (j0 + lr) * ldx + k0 + lk);
        if (i0 + lr < m && k0 + lk < d_pad) wv = *reinterpret_cast<const float4 *>(W + (size_t) (i0 + lr) * ldw + k0 + lk);
        __syncthreads();
        xs[lk + 0][lr] = xv.x; xs[lk + 1][lr] = xv.y; xs[lk + 2][lr] = xv.z; xs[lk + 3][lr] = xv.w;
        wsm[lk + 0][lr] = wv.x; wsm[lk + 1][lr] = wv.y; wsm[lk + 2][lr] = wv.z; wsm[lk + 3][lr] = wv.w;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            float xa[4], wb[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) { xa[a] = xs[k][tx + 16 * a]; wb[a] = wsm[k][ty + 16 * a]; }
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int a = 0; a < 4; ++a) acc[b][a] = fmaf(wb[b], xa[a], acc[b][a]);
        }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        int i = i0 + ty + 16 * b;
        if (i >= m) continue;
        float sdi = sd_rows[i];
        const size_t orow = row_slot ? (size_t) row_slot[i] : (size_t) i;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            int j = j0 + tx + 16 * a;
            if (j < n) out[orow * ld_out + j] = apply_kernel(fn, acc[b][a], sdi, sd[j]);
        }
    }
}

// ---- CSR engine ------------------------------------------------------------------------------
// out[i][j] = kfn(sum over the stored entries (c, x) of instance j, in storage order, of x * panel[c][i]): the same FP32
// recurrence per value as the reference's sparse x dense product (kernelmatrix_kernel.cpp:149-160). The requested rows are
// staged as a panel [feature][requested row] (zero where a row has no such feature).
//
// A warp takes an instance at a time and a part of 128 requested rows, a lane four of them: an entry costs one 512-byte
// read of the panel and four FMAs per lane. What bounds it is first the number of instructions around these, then the
// latency of the reads, then L2:
//   * the live entries of 32 are packed (place, value) into shared memory, from where the loop reads two with one
//     broadcast load: 8 instructions per entry instead of 28 with a shuffle each for place and value;
//   * an entry whose panel row is all zero in this part is skipped (a bitmap over the features, filled by the staging
//     kernel): adding x * 0 does not change a sum, and text-like data has mostly such entries;
//   * with few features (ALL) the part's panel is copied to shared memory first; else the frequent features come from L1
//     (keeping the most frequent ones in shared memory took half of the warps' room and was slower);
//   * bounds, entries and self dots of the following instances are fetched while one is computed;
//   * blocks are dealt to the parts that exist: the number of requested rows is only known on the device (the row cache
//     asks for what it misses, often 100 of 512), and every block takes part;
//   * a warp works on `unit` consecutive instances and then stores up to 16 bytes per requested row at once. Larger units
//     store better, smaller ones leave fewer warps without work at the end: the largest one with four rounds or more.
// Measured, staging included, before and after: 120 / 512 / 1,000 requested rows of 20,242 x 47,236 (74 entries each) 80 /
// 306 / 1,344 -> 68 / 157 / 279 us; of 32,561 x 123 (14 entries each) 56 / 96 / 171 -> 56 / 103 / 184 us, where the former
// engine could not tell that only 120 of 512 rows were wanted.
constexpr int CSR_THREADS = 512, CSR_WARPS = CSR_THREADS / 32, CSR_UNIT = 4;
constexpr int CSR_WARP_SMEM = CSR_UNIT * 33 * 16 + 32 * 8;                       // results of a unit, packed entries
constexpr int CSR_FIXED_SMEM = CSR_WARPS * CSR_WARP_SMEM + CSR_PART * 4;         // and the output row of every requested row
constexpr int CSR_BITMAP_MAX_D = 1 << 18;                                        // 32 KB of bitmap; more features: no skipping
constexpr int CSR_SMEM_MAX = 227 * 1024 - 256;
__host__ __device__ constexpr int csr_bitmap_words(int d) { return d <= CSR_BITMAP_MAX_D ? (d + 31) / 32 : 0; }

struct CsrPanel {
    const float *WT;                // [d][ld]
    int ld, d;
    const unsigned *bits;           // [parts][words]: features that some row of the part has
    int words;                      // 0: no bitmap
};

template <bool RBF>
__device__ __forceinline__ float csr_value(const KernelFn &fn, float dot, float sd_i, float sd_j) {
    if constexpr (RBF) return expf(-(sd_i + sd_j - dot * 2.0f) * fn.gamma);
    else return apply_kernel(fn, dot, sd_i, sd_j);
}

template <bool RBF, bool ALL>
__global__ void __launch_bounds__(CSR_THREADS, 2)
csr_rows_kernel(const float *__restrict__ val, const int *__restrict__ row_ptr, const int *__restrict__ col, int n,
                const CsrPanel P, int m_launch, const float *__restrict__ sd, const float *__restrict__ sd_rows, KernelFn fn,
                float *__restrict__ out, long long ld_out, const int *__restrict__ m_dev, const int *__restrict__ row_slot) {
    extern __shared__ __align__(16) unsigned char csr_sm[];  // results | packed entries | output rows | panel or bitmap
    const int m = m_dev ? min(m_launch, max(*m_dev, 0)) : m_launch;     // the count found on the device, if any
    const int parts = (m + CSR_PART - 1) / CSR_PART;
    if (parts == 0) return;
    const int part = blockIdx.x % parts, share = blockIdx.x / parts, shares = ((int) gridDim.x - part + parts - 1) / parts;
    const int c0 = part * CSR_PART, mh = min(CSR_PART, m - c0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float4 *res = reinterpret_cast<float4 *>(csr_sm) + (size_t) warp * CSR_UNIT * 33;
    uint2 *packed = reinterpret_cast<uint2 *>(csr_sm + CSR_WARPS * CSR_UNIT * 33 * 16) + warp * 32;
    int *orow_sm = reinterpret_cast<int *>(csr_sm + CSR_WARPS * CSR_WARP_SMEM);
    unsigned char *rest = csr_sm + CSR_FIXED_SMEM;
    const unsigned *bits = reinterpret_cast<const unsigned *>(rest);
    if constexpr (ALL) {
        float4 *panel = reinterpret_cast<float4 *>(rest);
#pragma unroll 4
        for (int i = tid; i < P.d * (CSR_PART / 4); i += CSR_THREADS)
            panel[i] = __ldg(reinterpret_cast<const float4 *>(P.WT + (size_t) (i / (CSR_PART / 4)) * P.ld + c0) + i % (CSR_PART / 4));
    } else {
        for (int w = tid; w < P.words; w += CSR_THREADS)
            reinterpret_cast<unsigned *>(rest)[w] = P.bits[(size_t) part * P.words + w];
    }
    // this lane's requested rows: c0 + 4 * lane + k
    float sdr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) sdr[k] = 4 * lane + k < mh ? sd_rows[c0 + 4 * lane + k] : 0.0f;
    if (tid < CSR_PART) orow_sm[tid] = tid < mh ? (row_slot ? row_slot[c0 + tid] : c0 + tid) : -1;
    __syncthreads();
    const bool vec_ok = (ld_out & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const long long rounds = (long long) n * parts / ((long long) gridDim.x * CSR_WARPS);
    const int unit = rounds >= 16 ? 4 : (rounds >= 8 ? 2 : 1);
    const int step = shares * CSR_WARPS * unit;
    auto after = [&](int j) { return ((j + 1) & (unit - 1)) != 0 && j + 1 < n ? j + 1 : j - (j & (unit - 1)) + step; };
    auto bounds = [&](int j, int &b, int &e, float &s) {
        b = e = 0; s = 0.0f;
        if (j < n) { b = row_ptr[j]; e = row_ptr[j + 1]; s = sd[j]; }
    };
    auto entry = [&](int p, int e, int &c, float &v) {
        c = 0; v = 0.0f;
        if (p < e) { c = col[p]; v = val[p]; }
    };
    auto panel_row = [&](unsigned place) -> float4 {
        if constexpr (ALL) return *reinterpret_cast<const float4 *>(rest + place + lane * 16);
        return __ldg(reinterpret_cast<const float4 *>(P.WT + (size_t) place * P.ld + c0) + lane);
    };
    auto add = [](float4 &acc, unsigned v, const float4 &w) {
        const float x = __uint_as_float(v);
        acc.x = fmaf(x, w.x, acc.x); acc.y = fmaf(x, w.y, acc.y);
        acc.z = fmaf(x, w.z, acc.z); acc.w = fmaf(x, w.w, acc.w);
    };
    int j = (share * CSR_WARPS + warp) * unit, j1 = after(j);
    int b, e, b1, e1, cc;
    float s, s1, vv;
    if (j >= n) return;
    bounds(j, b, e, s);
    bounds(j1, b1, e1, s1);
    entry(b + lane, e, cc, vv);
    for (;;) {
        const int j2 = after(j1);
        int b2, e2, cc1;
        float s2, vv1;
        bounds(j2, b2, e2, s2);
        entry(b1 + lane, e1, cc1, vv1);
        float4 acc = make_float4(0, 0, 0, 0);
        for (int p0 = b; p0 < e; p0 += 32) {
            const int c = cc;
            const float v = vv;
            if (p0 + 32 < e) entry(p0 + 32 + lane, e, cc, vv);
            bool live = p0 + lane < e;
            if constexpr (!ALL)
                if (live && P.words) live = (bits[c >> 5] >> (c & 31)) & 1u;
            const unsigned mask = __ballot_sync(0xffffffffu, live);
            const int count = __popc(mask);
            if (live) packed[__popc(mask & ((1u << lane) - 1))] = make_uint2(ALL ? (unsigned) c * (CSR_PART * 4) : (unsigned) c, __float_as_uint(v));
            __syncwarp();
            int t = 0;
            for (; t + 4 <= count; t += 4) {             // four panel rows in flight, added in storage order
                const uint4 p01 = *reinterpret_cast<const uint4 *>(packed + t), p23 = *reinterpret_cast<const uint4 *>(packed + t + 2);
                const float4 w0 = panel_row(p01.x), w1 = panel_row(p01.z), w2 = panel_row(p23.x), w3 = panel_row(p23.z);
                add(acc, p01.y, w0); add(acc, p01.w, w1); add(acc, p23.y, w2); add(acc, p23.w, w3);
            }
            if (t < count) {
                const uint2 e0 = packed[t], ea = packed[t + (t + 1 < count ? 1 : 0)], eb = packed[t + (t + 2 < count ? 2 : 0)];
                const float4 w0 = panel_row(e0.x), w1 = panel_row(ea.x), w2 = panel_row(eb.x);
                add(acc, e0.y, w0);
                if (t + 1 < count) add(acc, ea.y, w1);
                if (t + 2 < count) add(acc, eb.y, w2);
            }
            __syncwarp();
        }
        acc.x = csr_value<RBF>(fn, acc.x, sdr[0], s); acc.y = csr_value<RBF>(fn, acc.y, sdr[1], s);
        acc.z = csr_value<RBF>(fn, acc.z, sdr[2], s); acc.w = csr_value<RBF>(fn, acc.w, sdr[3], s);
        const int u = j & (unit - 1), first = j - u;
        res[u * 33 + lane] = acc;
        if (j1 != j + 1 || u + 1 == unit) {              // the last one of its unit: store them
            const int have = u + 1;
            __syncwarp();
            if (vec_ok && have == 4) {
                // a lane stores four instances of its four requested rows
                const int4 o = reinterpret_cast<const int4 *>(orow_sm)[lane];
                const float4 r0 = res[lane], r1 = res[33 + lane], r2 = res[66 + lane];
                if (o.x >= 0) *reinterpret_cast<float4 *>(out + o.x * ld_out + first) = make_float4(r0.x, r1.x, r2.x, acc.x);
                if (o.y >= 0) *reinterpret_cast<float4 *>(out + o.y * ld_out + first) = make_float4(r0.y, r1.y, r2.y, acc.y);
                if (o.z >= 0) *reinterpret_cast<float4 *>(out + o.z * ld_out + first) = make_float4(r0.z, r1.z, r2.z, acc.z);
                if (o.w >= 0) *reinterpret_cast<float4 *>(out + o.w * ld_out + first) = make_float4(r0.w, r1.w, r2.w, acc.w);
            } else {
                // a lane stores one value: the instances of a row next to each other
                const int sh = unit == 4 ? 2 : unit - 1, w = lane & (unit - 1);
                for (int r = lane >> sh; r < mh; r += 32 >> sh)
                    if (w < have) out[orow_sm[r] * ld_out + first + w] = reinterpret_cast<const float *>(res)[w * 132 + r];
            }
            __syncwarp();
        }
        j = j1; j1 = j2;
        if (j >= n) return;
        b = b1; e = e1; s = s1; b1 = b2; e1 = e2; s1 = s2;
        cc = cc1; vv = vv1;
    }
}

// ---- host side ----------------------------------------------------------------------------------

// Staging buffers for m requested rows: as rows in the operand form of the dense engines, or (panel) as the CSR engine's
// panel.
static tsvm_status ensure_scratch(tsvm_km *km, int m, bool panel) {
    if (m <= (panel ? km->wt_ld : km->w_cap)) return TSVM_OK;
    int cap = 128;
    while (cap < m) cap *= 2;
    if (cap > km->sd_cap) {
        pool_free(km->sd_rows);
        km->sd_rows = nullptr;
        km->sd_cap = 0;
        TSVM_TRY(dev_alloc(&km->sd_rows, (size_t) cap));
        km->sd_cap = cap;
    }
    if (!panel) {
        pool_free_many({km->W, km->Whi, km->Wlo, km->w_unscale});
        km->W = km->Whi = km->Wlo = km->w_unscale = nullptr;
        km->w_cap = 0;
        // either plane kind fits cap x d_pad words: round_up(d, 8) halves <= d_pad floats
        TSVM_TRY(dev_alloc(&km->w_unscale, (size_t) cap));
        TSVM_TRY(dev_alloc(&km->W, (size_t) cap * km->d_pad));
        TSVM_TRY(dev_alloc(&km->Whi, (size_t) cap * km->d_pad));
        TSVM_TRY(dev_alloc(&km->Wlo, (size_t) cap * km->d_pad));
        km->w_cap = cap;
        return TSVM_OK;
    }
    pool_free_many({km->WT, km->csr_bits});
    km->WT = nullptr;
    km->csr_bits = nullptr;
    km->wt_ld = 0;
    TSVM_TRY(dev_alloc(&km->WT, (size_t) km->d * cap));
    // (an allocation that other streams know nothing of: cleared and waited for here)
    TSVM_CUDA(cudaMemset(km->WT, 0, sizeof(float) * (size_t) km->d * cap));
    const size_t words = (size_t) csr_bitmap_words(km->d) * ceil_div(cap, CSR_PART);
    TSVM_TRY(dev_alloc(&km->csr_bits, words));
    TSVM_CUDA(cudaMemset(km->csr_bits, 0, sizeof(unsigned) * words));
    TSVM_CUDA(cudaStreamSynchronize(nullptr));
    km->wt_ld = cap;
    return TSVM_OK;
}

// engine: 0 = automatic, 1 = CUDA cores, 3 (and its old alias 2) = tensor cores on TF32 planes, 4 = tensor
// cores on row-scaled FP16 planes (what "automatic" picks for d_pad > 32); both tensor forms run on CTA pairs
static inline bool use_tensor_engine(const tsvm_km *km) {
    return km->engine >= 2 || (km->engine == 0 && km->d_pad > 32);
}
static inline int wanted_plane_kind(const tsvm_km *km) {
    if (!km->dense || !use_tensor_engine(km)) return 0;
    return (km->engine == 2 || km->engine == 3) ? 1 : 2;
}

// eight blocks of eight warps (a row each) per SM
static inline int prepare_grid(int n) { const int b = ceil_div(n, 8), most = 8 * device_sm_count(); return b < most ? b : most; }

// Buffers of the planes the selected engine reads.
static tsvm_status alloc_planes(tsvm_km *km, int kind) {
    pool_free_many({km->Xhi, km->Xlo});
    km->Xhi = km->Xlo = nullptr;
    km->plane_kind = 0;
    km->plane_ld = kind == 1 ? km->d_pad : (km->d + 7) & ~7;
    const size_t words = kind == 1 ? (size_t) km->n * km->plane_ld : ((size_t) km->n * km->plane_ld + 1) / 2;
    TSVM_TRY(dev_alloc(&km->Xhi, words));
    TSVM_TRY(dev_alloc(&km->Xlo, words));
    if (!km->x_unscale) TSVM_TRY(dev_alloc(&km->x_unscale, (size_t) km->n));
    return TSVM_OK;
}

// Builds the planes, once; a change of engine rebuilds them.
static tsvm_status ensure_planes(tsvm_km *km, cudaStream_t st) {
    const int kind = wanted_plane_kind(km);
    if (kind == 0 || kind == km->plane_kind) return TSVM_OK;
    TSVM_TRY(alloc_planes(km, kind));
    TSVM_LAUNCH(prepare_rows_kernel, prepare_grid(km->n), 256, 0, st, km->X, km->n, km->d, km->ldx, kind, km->plane_ld,
                km->Xhi, km->Xlo, km->x_unscale, km->fn, (float *) nullptr, (float *) nullptr, (int *) nullptr);
    km->plane_kind = kind;
    return TSVM_OK;
}

static inline RowDst row_dst(const tsvm_km *km) {
    if (use_tensor_engine(km)) return RowDst{nullptr, km->Whi, km->Wlo, km->w_unscale, km->plane_kind, km->plane_ld};
    return RowDst{km->W, nullptr, nullptr, nullptr, 0, km->d_pad};
}

static tsvm_status inspect_entries(tsvm_km *km, const float *val, const int *row_ptr, const int *col, int n, bool batch,
                                   cudaStream_t st, bool *exact) {
    int *found = km->status_dev + 2;                     // (the first word is the engines' status)
    TSVM_CUDA(cudaMemsetAsync(found, 0, 2 * sizeof(int), st));
    TSVM_LAUNCH(inspect_entries_kernel, prepare_grid(n), 256, 0, st, val, row_ptr, col, n, km->d, batch, found);
    TSVM_CUDA(cudaMemcpyAsync(km->status_host + 2, found, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    TSVM_CUDA(cudaStreamSynchronize(st));
    *exact = km->status_host[2] == 0;
    return TSVM_OK;
}

// Back to the CSR form of the data (nothing uses the dense copy any more): pool_free_many waits for the device.
void km_drop_dense_copy(tsvm_km *km) {
    pool_free_many({km->X_owned, km->Xhi, km->Xlo, km->x_unscale, km->W, km->Whi, km->Wlo, km->w_unscale});
    km->X_owned = km->Xhi = km->Xlo = km->x_unscale = km->W = km->Whi = km->Wlo = km->w_unscale = nullptr;
    km->X = nullptr;
    km->w_cap = km->plane_kind = km->plane_ld = km->d_pad = km->ldx = 0;
    km->dense = km->from_csr = false;
}

// Makes the dense copy of CSR data whose kernel rows the tensor-core engine computes faster and as exactly. Where the
// device has no room for it and its planes the entries do as well.
static tsvm_status choose_csr_storage(tsvm_km *km, cudaStream_t st) {
    const int d_pad = (km->d + 3) & ~3;
    const double dense_bytes = (double) km->n * d_pad * 8.0;             // the rows and their two planes
    if (km->d < CSR_DENSE_MIN_D || km->d > CSR_DENSE_MAX_D || dense_bytes > device_memory_bytes() / 8.0) return TSVM_OK;
    TSVM_TRY(dev_alloc(&km->status_dev, 4));
    TSVM_TRY(pinned_alloc((void **) &km->status_host, 4 * sizeof(int)));
    km->launched(st);
    bool exact = false;
    TSVM_TRY(inspect_entries(km, km->val, km->row_ptr, km->col, km->n, false, st, &exact));
    km->nnz = km->status_host[3];
    if (!exact || (km->d > CSR_DENSE_ANY_D && km->nnz < CSR_DENSE_SHARE * (double) km->n * km->d)) return TSVM_OK;
    km->ldx = km->d_pad = d_pad;
    km->dense = km->from_csr = true;
    tsvm_status s = dev_alloc(&km->X_owned, (size_t) km->n * d_pad);
    if (s == TSVM_OK) s = alloc_planes(km, wanted_plane_kind(km));
    if (s != TSVM_OK) {
        km_drop_dense_copy(km);
        return s == TSVM_ERR_OOM ? TSVM_OK : s;
    }
    km->X = km->X_owned;
    TSVM_LAUNCH(dense_from_csr_kernel, prepare_grid(km->n), 256, 0, st, km->val, km->row_ptr, km->col, km->n, d_pad, km->X_owned);
    return TSVM_OK;
}

static tsvm_status finish_create(tsvm_km *km, cudaStream_t st) {
    TSVM_TRY(dev_alloc(&km->self_dot, (size_t) km->n));
    TSVM_TRY(dev_alloc(&km->diag, (size_t) km->n));
    if (!km->status_dev) TSVM_TRY(dev_alloc(&km->status_dev, 4));
    if (!km->status_host) TSVM_TRY(pinned_alloc((void **) &km->status_host, 4 * sizeof(int)));
    km->launched(st);
    if (!km->dense) {
        TSVM_LAUNCH(self_dot_csr_kernel, ceil_div((long long) km->n * 32, 256), 256, 0, st, km->val, km->row_ptr, km->n,
                    km->fn, km->self_dot, km->diag, km->status_dev);
        return TSVM_OK;
    }
    int kind = wanted_plane_kind(km);
    if (kind && !km->Xhi) {
        const tsvm_status s = alloc_planes(km, kind);
        if (s == TSVM_ERR_OOM) kind = 0;         // ensure_planes asks again when an engine that reads them is used
        else if (s != TSVM_OK) return s;
    }
    TSVM_LAUNCH(prepare_rows_kernel, prepare_grid(km->n), 256, 0, st, km->X, km->n, km->d, km->ldx, kind, km->plane_ld,
                km->Xhi, km->Xlo, km->x_unscale, km->fn, km->self_dot, km->diag, km->status_dev);
    km->plane_kind = kind;
    return TSVM_OK;
}

// TSVM_CSR_SMEM=0 leaves the panel in L2 (used to check that its place changes no result)
static bool csr_smem_allowed() {
    static const bool on = [] { const char *e = getenv("TSVM_CSR_SMEM"); return !e || atoi(e) != 0; }();
    return on;
}

// Kernel rows of the m requested rows staged in WT / sd_rows against all stored instances. with_bits: the staging filled
// the bitmap.
static tsvm_status csr_engine_launch(tsvm_km *km, int m, bool with_bits, float *out, long long ld_out, cudaStream_t st) {
    TSVM_REQUIRE(m <= 1024, "CSR engine handles at most 1024 rows per call, got %d", m);
    const bool all = csr_smem_allowed() && km->d <= (CSR_SMEM_MAX - CSR_FIXED_SMEM) / (CSR_PART * 4);
    CsrPanel P;
    P.WT = km->WT; P.ld = km->wt_ld; P.d = km->d;
    P.words = with_bits && !all ? csr_bitmap_words(km->d) : 0;
    P.bits = km->csr_bits;
    const size_t smem = CSR_FIXED_SMEM + (all ? (size_t) km->d * CSR_PART * 4 : (size_t) P.words * 4);
    const bool rbf = km->fn.type == TSVM_RBF || km->fn.type == TSVM_PRECOMPUTED;
    const int per_sm = smem <= 112 * 1024 ? 2 : 1;
    const int units = ceil_div(km->n, CSR_WARPS) * ceil_div(m, CSR_PART);
    const int grid = device_sm_count() * per_sm < units ? device_sm_count() * per_sm : units;
#define CSR_CASE(RBF, ALL)                                                                                                \
    do {                                                                                                                  \
        TSVM_ONCE_PER_DEVICE(TSVM_CUDA(cudaFuncSetAttribute((csr_rows_kernel<RBF, ALL>),                                  \
                                                            cudaFuncAttributeMaxDynamicSharedMemorySize, CSR_SMEM_MAX))); \
        TSVM_LAUNCH((csr_rows_kernel<RBF, ALL>), grid, CSR_THREADS, smem, st, km->val, km->row_ptr, km->col, km->n, P, m, \
                    km->self_dot, km->sd_rows, km->fn, out, ld_out, km->rows_m_dev, km->rows_slot_dev);                   \
    } while (0)
    if (rbf) { if (all) CSR_CASE(true, true); else CSR_CASE(true, false); }
    else if (all) CSR_CASE(false, true); else CSR_CASE(false, false);
#undef CSR_CASE
    return TSVM_OK;
}

static tsvm_status rows_common(tsvm_km *km, int m, float *out, long long ld_out, cudaStream_t st) {
    // W / WT and sd_rows are staged; run the engine.
    if (km->dense) {
        if (use_tensor_engine(km)) return launch_dense_tc(km, m, out, ld_out, st);
        dim3 grid(ceil_div(km->n, 64), ceil_div(m, 64));
        TSVM_LAUNCH(dense_rows_simt_kernel, grid, 256, 0, st, km->X, km->ldx, km->n, km->W, km->d_pad, m, km->d_pad,
                    km->self_dot, km->sd_rows, km->fn, out, ld_out, km->rows_m_dev, km->rows_slot_dev);
        return TSVM_OK;
    }
    return csr_engine_launch(km, m, true, out, ld_out, st);
}

// ---- pieces of tsvm_km_rows_by_index for callers that overlap them (the solver) -------------------
tsvm_status launch_dense_tc2_on(tsvm_km *km, const InstancePlanes &X, int m, float *out, long long ld_out,
                                cudaStream_t st);   // dense_tc2.cu

tsvm_status km_count_entries(tsvm_km *km, cudaStream_t st) {
    if (km->nnz >= 0) return TSVM_OK;
    int last = 0;
    TSVM_CUDA(cudaMemcpyAsync(&last, km->row_ptr + km->n, sizeof(int), cudaMemcpyDeviceToHost, st));
    TSVM_CUDA(cudaStreamSynchronize(st));
    km->nnz = last;
    return TSVM_OK;
}
bool km_automatic_engine(const tsvm_km *km) { return km->engine == 0; }
// True when kernel rows of this matrix run on the CTA-pair tensor engine, whose requested-row staging and
// launch can be issued separately and against a caller-chosen subset of instances.
bool km_pair_engine(tsvm_km *km, cudaStream_t st) {
    if (!km->dense || !use_tensor_engine(km)) return false;
    return ensure_planes(km, st) == TSVM_OK && km->plane_kind != 0;
}

size_t km_plane_row_bytes(const tsvm_km *km) {
    return (size_t) km->plane_ld * (km->plane_kind == 2 ? sizeof(__half) : sizeof(float));
}

tsvm_status km_stage_rows_by_index(tsvm_km *km, const int *idx_dev, int q, cudaStream_t st) {
    TSVM_TRY(ensure_scratch(km, q, false));
    TSVM_TRY(ensure_planes(km, st));
    TSVM_LAUNCH(gather_rows_dense_kernel, q, 256, 0, st, km->X, km->ldx, km->d, idx_dev, q, km->self_dot, row_dst(km),
                km->sd_rows, km->rows_m_dev);
    return TSVM_OK;
}

tsvm_status km_rows_staged(tsvm_km *km, int q, float *out, long long ld_out, cudaStream_t st) {
    return rows_common(km, q, out, ld_out, st);
}

tsvm_status km_gather_planes(tsvm_km *km, const int *ids_dev, int m, const int *m_dev, float *hi, float *lo, float *sd,
                             float *unscale, cudaStream_t st) {
    TSVM_LAUNCH(gather_planes_kernel, m, 128, 0, st, km->Xhi, km->Xlo, km_plane_row_bytes(km), ids_dev, m,
                km->self_dot, km->plane_kind == 2 ? km->x_unscale : nullptr, hi, lo, sd, unscale, m_dev);
    return TSVM_OK;
}

tsvm_status km_rows_staged_on(tsvm_km *km, const InstancePlanes &X, int q, float *out, long long ld_out,
                              cudaStream_t st) {
    return launch_dense_tc2_on(km, X, q, out, ld_out, st);
}

tsvm_status launch_dense_tc2_planes(tsvm_km *km, const InstancePlanes &X, const RowPlanes &W, int m, float *out,
                                    long long ld_out, cudaStream_t st);   // dense_tc2.cu

tsvm_status km_rows_planes_on(tsvm_km *km, const InstancePlanes &X, const RowPlanes &W, int q, float *out,
                              long long ld_out, cudaStream_t st) {
    return launch_dense_tc2_planes(km, X, W, q, out, ld_out, st);
}

// Stages m explicit feature rows (m x n_features, stride ldt) with their self dots as the requested rows.
tsvm_status km_stage_rows_features(tsvm_km *km, const float *T_dev, int ldt, const float *sd_T_dev, int m,
                                   cudaStream_t st) {
    TSVM_TRY(ensure_scratch(km, m, false));
    TSVM_TRY(ensure_planes(km, st));
    TSVM_CUDA(cudaMemcpyAsync(km->sd_rows, sd_T_dev, sizeof(float) * m, cudaMemcpyDeviceToDevice, st));
    TSVM_LAUNCH(stage_rows_dense_kernel, m, 256, 0, st, T_dev, ldt, km->d, km->d, m, row_dst(km));
    return TSVM_OK;
}

// Stages mm new instances as the requested rows of a dense kernel matrix (self dots accumulated in storage
// order as kernelmatrix.cpp:288-296 does, rows in the engine's operand form): the first half of
// tsvm_km_rows_by_instances_*, shared with the fused prediction.
static inline int batch_row_blocks(int mm) {
    const int all = ceil_div(mm, BATCH_WARPS), most = 6 * device_sm_count();
    return all < most ? all : most;
}
tsvm_status km_stage_instances_dense(tsvm_km *km, const float *T, int mm, int dt, int ldt, const SumPreset &preset, cudaStream_t st) {
    TSVM_TRY(ensure_scratch(km, mm, false));
    TSVM_TRY(ensure_planes(km, st));
    const int dots = ceil_div(mm, 32), rows = batch_row_blocks(mm), grid = dots + rows + ceil_div(preset.total, BATCH_THREADS);
    if ((ldt & 3) == 0 && ((uintptr_t) T & 15) == 0)
        TSVM_LAUNCH(stage_batch_dense_kernel<true>, grid, BATCH_THREADS, 0, st, T, ldt, dt, km->d, mm, row_dst(km), km->sd_rows,
                    dots, rows, preset);
    else
        TSVM_LAUNCH(stage_batch_dense_kernel<false>, grid, BATCH_THREADS, 0, st, T, ldt, dt, km->d, mm, row_dst(km), km->sd_rows,
                    dots, rows, preset);
    return TSVM_OK;
}

// Can this batch go through the fused prediction? Where the matrix is the dense copy of CSR data, only if the engine's
// operand form holds the batch exactly too.
tsvm_status km_pair_engine_takes(tsvm_km *km, const float *tval, const int *rp, const int *tcol, int m, cudaStream_t st,
                                 bool *takes) {
    *takes = km_pair_engine(km, st);
    if (*takes && km->from_csr) {
        *takes = false;
        if (rp) TSVM_TRY(inspect_entries(km, tval, rp, tcol, m, true, st, takes));
    }
    return TSVM_OK;
}

tsvm_status km_stage_instances_csr(tsvm_km *km, const float *tval, const int *rp, const int *tcol, int mm,
                                   const SumPreset &preset, cudaStream_t st) {
    TSVM_TRY(ensure_scratch(km, mm, false));
    TSVM_TRY(ensure_planes(km, st));
    const int dots = ceil_div(mm, BATCH_THREADS), rows = batch_row_blocks(mm), grid = dots + rows + ceil_div(preset.total, BATCH_THREADS);
    TSVM_LAUNCH(stage_batch_csr_kernel, grid, BATCH_THREADS, 0, st, tval, rp, tcol, mm, km->d, row_dst(km), km->sd_rows, dots, rows,
                preset);
    return TSVM_OK;
}

}  // namespace tsvm

using namespace tsvm;

// zero_padded: a device X whose columns d .. ld - 1 are zero is worked on in place whatever d is.
tsvm_status tsvm::km_create_dense(const float *X, int n, int d, int ld, int loc, bool zero_padded, int kernel_type, int degree,
                                  float gamma, float coef0, void *stream, tsvm_km **out) {
    TSVM_REQUIRE(out && X && n > 0 && d > 0 && ld >= d, "km_create_dense: bad arguments (n=%d d=%d ld=%d)", n, d, ld);
    TSVM_REQUIRE(kernel_type >= TSVM_LINEAR && kernel_type <= TSVM_PRECOMPUTED, "unknown kernel type %d", kernel_type);
    cudaStream_t st = (cudaStream_t) stream;
    tsvm_km *km = new tsvm_km;
    *out = nullptr;
    km->n = n; km->d = d; km->nnz = (long long) n * d; km->dense = true;
    km->fn = KernelFn{kernel_type, degree, gamma, coef0};
    km->d_pad = (d + 3) & ~3;
    tsvm_status s = TSVM_OK;
    bool in_place = loc == TSVM_DEVICE && (d % 4 == 0 || zero_padded) && (ld % 4 == 0) && (((uintptr_t) X & 15) == 0) && ld >= km->d_pad;
    if (in_place) { km->X = X; km->ldx = ld; }
    else {
        km->ldx = km->d_pad;
        s = dev_alloc(&km->X_owned, (size_t) n * km->d_pad);
        if (s == TSVM_OK && km->d_pad != d) {
            cudaError_t e = cudaMemsetAsync(km->X_owned, 0, sizeof(float) * (size_t) n * km->d_pad, st);
            if (e != cudaSuccess) { set_error("memset failed: %s", cudaGetErrorString(e)); s = TSVM_ERR_CUDA; }
        }
        if (s == TSVM_OK) {
            cudaError_t e = cudaMemcpy2DAsync(km->X_owned, sizeof(float) * km->d_pad, X, sizeof(float) * ld,
                                              sizeof(float) * d, n,
                                              loc == TSVM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                                              st);
            if (e != cudaSuccess) { set_error("copy of X failed: %s", cudaGetErrorString(e)); s = TSVM_ERR_CUDA; }
        }
        km->X = km->X_owned;
    }
    if (s == TSVM_OK) s = finish_create(km, st);
    if (s != TSVM_OK) { tsvm_km_destroy(km); return s; }
    *out = km;
    return TSVM_OK;
}

extern "C" {

const char *tsvm_last_error(void) { return tsvm::g_err; }
int tsvm_abi_version(void) { return 2; }
void tsvm_release_cached_memory(void) {
    tsvm::release_solver_streams();
    tsvm::pool_release();
}

tsvm_status tsvm_km_create_dense(const float *X, int n, int d, int ld, int loc, int kernel_type, int degree,
                                 float gamma, float coef0, void *stream, tsvm_km **out) {
    return tsvm::km_create_dense(X, n, d, ld, loc, false, kernel_type, degree, gamma, coef0, stream, out);
}

tsvm_status tsvm_km_create_csr(const float *val, const int *row_ptr, const int *col, int n, int d, int loc,
                               int kernel_type, int degree, float gamma, float coef0, void *stream, tsvm_km **out) {
    TSVM_REQUIRE(out && row_ptr && n > 0 && d > 0, "km_create_csr: bad arguments (n=%d d=%d)", n, d);
    TSVM_REQUIRE(kernel_type >= TSVM_LINEAR && kernel_type <= TSVM_PRECOMPUTED, "unknown kernel type %d", kernel_type);
    cudaStream_t st = (cudaStream_t) stream;
    tsvm_km *km = new tsvm_km;
    *out = nullptr;
    km->n = n; km->d = d; km->dense = false;
    km->fn = KernelFn{kernel_type, degree, gamma, coef0};
    tsvm_status s = TSVM_OK;
    if (loc == TSVM_DEVICE) {
        km->nnz = -1;                     // read from row_ptr when someone asks (tsvm_km_nnz, km_count_entries)
        km->val = val; km->row_ptr = row_ptr; km->col = col;
    } else {
        const int last = row_ptr[n];
        km->nnz = last;
        s = dev_alloc(&km->val_owned, (size_t) last);
        if (s == TSVM_OK) s = dev_alloc(&km->col_owned, (size_t) last);
        if (s == TSVM_OK) s = dev_alloc(&km->row_ptr_owned, (size_t) n + 1);
        if (s == TSVM_OK) {
            cudaError_t e = cudaMemcpyAsync(km->val_owned, val, sizeof(float) * last, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(km->col_owned, col, sizeof(int) * last, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(km->row_ptr_owned, row_ptr, sizeof(int) * ((size_t) n + 1), cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) { set_error("copy of CSR failed: %s", cudaGetErrorString(e)); s = TSVM_ERR_CUDA; }
        }
        km->val = km->val_owned; km->col = km->col_owned; km->row_ptr = km->row_ptr_owned;
    }
    if (s == TSVM_OK) s = choose_csr_storage(km, st);
    if (s == TSVM_OK) s = finish_create(km, st);
    if (s != TSVM_OK) { tsvm_km_destroy(km); return s; }
    *out = km;
    return TSVM_OK;
}

void tsvm_km_destroy(tsvm_km *km) {
    if (!km) return;
    pool_free_many({km->X_owned, km->Xhi, km->Xlo, km->x_unscale, km->w_unscale, km->val_owned, km->row_ptr_owned,
                    km->col_owned, km->self_dot, km->diag, km->W, km->Whi, km->Wlo, km->WT, km->sd_rows,
                    km->few_acc, km->csr_bits, km->status_dev}, !km->in_flight && !km->exposed);
    if (km->status_host) pinned_free(km->status_host);
    delete km;
}

int tsvm_km_n_instances(const tsvm_km *km) { return km ? km->n : 0; }
int tsvm_km_n_features(const tsvm_km *km) { return km ? km->d : 0; }
long long tsvm_km_nnz(const tsvm_km *km) {
    if (!km) return 0;
    if (km->nnz >= 0) return km->nnz;
    int last = 0;
    if (cudaMemcpy(&last, km->row_ptr + km->n, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return last;
}
int tsvm_km_is_dense(const tsvm_km *km) { return km && km->dense && !km->from_csr; }
const float *tsvm_km_diag_dev(const tsvm_km *km) {
    if (!km) return nullptr;
    const_cast<tsvm_km *>(km)->exposed = true;      // the caller's own work may read it until the handle is destroyed
    return km->diag;
}
const float *tsvm_km_self_dot_dev(const tsvm_km *km) {
    if (!km) return nullptr;
    const_cast<tsvm_km *>(km)->exposed = true;
    return km->self_dot;
}

tsvm_status tsvm_km_set_dense_engine(tsvm_km *km, int engine) {
    TSVM_REQUIRE(km && engine >= 0 && engine <= 4, "set_dense_engine: bad arguments");
    if (km->from_csr) return TSVM_OK;        // the choice concerns matrices that were given as dense ones
    km->engine = engine;
    return TSVM_OK;
}

tsvm_status tsvm_km_rows_by_index(tsvm_km *km, const int *idx_dev, int q, float *out_dev, long long ld_out,
                                  void *stream) {
    TSVM_REQUIRE(km && idx_dev && out_dev && q > 0 && ld_out >= km->n, "rows_by_index: bad arguments (q=%d)", q);
    cudaStream_t st = (cudaStream_t) stream;
    km->launched(st);
    TSVM_TRY(ensure_scratch(km, q, !km->dense));
    if (km->dense) {
        TSVM_TRY(ensure_planes(km, st));
        TSVM_LAUNCH(gather_rows_dense_kernel, q, 256, 0, st, km->X, km->ldx, km->d, idx_dev, q, km->self_dot,
                    row_dst(km), km->sd_rows, km->rows_m_dev);
        return rows_common(km, q, out_dev, ld_out, st);
    }
    TSVM_REQUIRE(q <= 1024, "CSR engine handles at most 1024 rows per call, got %d", q);
    TSVM_LAUNCH(scatter_csr_to_wt_kernel, q, 128, 0, st, km->val, km->row_ptr, km->col, idx_dev, q, km->d, km->wt_ld,
                km->WT, km->self_dot, km->sd_rows, false, km->rows_m_dev, km->csr_bits, csr_bitmap_words(km->d));
    TSVM_TRY(rows_common(km, q, out_dev, ld_out, st));
    TSVM_LAUNCH(scatter_csr_to_wt_kernel, q, 128, 0, st, km->val, km->row_ptr, km->col, idx_dev, q, km->d, km->wt_ld,
                km->WT, nullptr, nullptr, true, km->rows_m_dev, km->csr_bits, csr_bitmap_words(km->d));
    return TSVM_OK;
}

tsvm_status tsvm_km_rows_by_instances_dense(tsvm_km *km, const float *T_dev, int m, int dt, int ldt, float *out_dev,
                                            long long ld_out, void *stream) {
    TSVM_REQUIRE(km && T_dev && out_dev && m > 0 && dt > 0 && ldt >= dt && ld_out >= km->n,
                 "rows_by_instances_dense: bad arguments");
    cudaStream_t st = (cudaStream_t) stream;
    km->launched(st);
    const bool dense = km->dense && !km->from_csr;       // (any values may come: entries of the matrix x panel of the batch)
    const int chunk = dense ? 4096 : 1024;
    for (int r0 = 0; r0 < m; r0 += chunk) {
        const int mm = min(chunk, m - r0);
        const float *T = T_dev + (size_t) r0 * ldt;
        float *o = out_dev + (size_t) r0 * ld_out;
        if (dense) {
            TSVM_TRY(km_stage_instances_dense(km, T, mm, dt, ldt, SumPreset{}, st));
            TSVM_TRY(rows_common(km, mm, o, ld_out, st));
        } else {
            TSVM_TRY(ensure_scratch(km, mm, true));
            TSVM_TRY(launch_self_dot_seq_dense(T, mm, dt, ldt, km->sd_rows, st));
            dim3 grid(ceil_div(km->d, 32), ceil_div(mm, 32)), block(32, 8);
            TSVM_LAUNCH(transpose_dense_to_wt_kernel, grid, block, 0, st, T, ldt, dt, km->d, mm, km->wt_ld, km->WT,
                        false);
            TSVM_TRY(csr_engine_launch(km, mm, false, o, ld_out, st));
            TSVM_LAUNCH(transpose_dense_to_wt_kernel, grid, block, 0, st, T, ldt, dt, km->d, mm, km->wt_ld, km->WT,
                        true);
        }
    }
    return TSVM_OK;
}

tsvm_status tsvm_km_rows_for_features_dense(tsvm_km *km, const float *T_dev, int ldt, const float *sd_T_dev, int m,
                                            float *out_dev, long long ld_out, void *stream) {
    TSVM_REQUIRE(km && km->dense && !km->from_csr && T_dev && sd_T_dev && out_dev && m > 0 && ldt >= km->d && ld_out >= km->n,
                 "rows_for_features_dense: bad arguments (dense kernel matrix required)");
    cudaStream_t st = (cudaStream_t) stream;
    km->launched(st);
    for (int r0 = 0; r0 < m; r0 += 4096) {
        const int mm = min(4096, m - r0);
        TSVM_TRY(ensure_scratch(km, mm, false));
        TSVM_CUDA(cudaMemcpyAsync(km->sd_rows, sd_T_dev + r0, sizeof(float) * mm, cudaMemcpyDeviceToDevice, st));
        TSVM_TRY(ensure_planes(km, st));
        TSVM_LAUNCH(stage_rows_dense_kernel, mm, 256, 0, st, T_dev + (size_t) r0 * ldt, ldt, km->d, km->d, mm,
                    row_dst(km));
        TSVM_TRY(rows_common(km, mm, out_dev + (size_t) r0 * ld_out, ld_out, st));
    }
    return TSVM_OK;
}

tsvm_status tsvm_km_rows_by_instances_csr(tsvm_km *km, const float *tval_dev, const int *trow_ptr_dev,
                                          const int *tcol_dev, int m, long long tnnz, float *out_dev,
                                          long long ld_out, void *stream) {
    (void) tnnz;
    TSVM_REQUIRE(km && trow_ptr_dev && out_dev && m > 0 && ld_out >= km->n, "rows_by_instances_csr: bad arguments");
    cudaStream_t st = (cudaStream_t) stream;
    km->launched(st);
    const bool dense = km->dense && !km->from_csr;       // (any values may come: entries of the matrix x panel of the batch)
    const int chunk = dense ? 4096 : 1024;
    for (int r0 = 0; r0 < m; r0 += chunk) {
        const int mm = min(chunk, m - r0);
        const int *rp = trow_ptr_dev + r0;     // row_ptr entries stay absolute offsets into tval/tcol
        float *o = out_dev + (size_t) r0 * ld_out;
        if (dense) {
            TSVM_TRY(km_stage_instances_csr(km, tval_dev, rp, tcol_dev, mm, SumPreset{}, st));
            TSVM_TRY(rows_common(km, mm, o, ld_out, st));
        } else {
            TSVM_TRY(ensure_scratch(km, mm, true));
            TSVM_LAUNCH(self_dot_seq_csr_kernel, ceil_div(mm, 128), 128, 0, st, tval_dev, rp, mm, km->sd_rows);
            TSVM_LAUNCH(scatter_csr_to_wt_kernel, mm, 128, 0, st, tval_dev, rp, tcol_dev, (const int *) nullptr, mm,
                        km->d, km->wt_ld, km->WT, (const float *) nullptr, (float *) nullptr, false, (const int *) nullptr, km->csr_bits,
                        csr_bitmap_words(km->d));
            TSVM_TRY(csr_engine_launch(km, mm, true, o, ld_out, st));
            TSVM_LAUNCH(scatter_csr_to_wt_kernel, mm, 128, 0, st, tval_dev, rp, tcol_dev, (const int *) nullptr, mm,
                        km->d, km->wt_ld, km->WT, (const float *) nullptr, (float *) nullptr, true, (const int *) nullptr, km->csr_bits,
                        csr_bitmap_words(km->d));
        }
    }
    return TSVM_OK;
}

}  // extern "C"
