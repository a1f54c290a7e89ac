// Decision values of a few test rows in one launch.
//
// A call with one row used to be seven launches and copies and two waits around 7 us of tensor-core work on a tile of 256
// rows (62 us per call at 3,001 x 100). Here the support vectors are read once, as they are stored, by blocks of warps
// that keep the test rows in shared memory; a block turns its dot products into kernel values, multiplies them by the
// coefficients, adds its sums to the decision values, and the last block of a row tile subtracts rho and votes.
//
// What bounds it: for few support vectors the chain of dependent memory trips (row -> barrier -> kernel value ->
// atomic -> ticket), about 8 us; for many the read of the support vectors (R = 1, 2) or the shared-memory reads of the
// test rows, R per four features (R = 8). Sums: FP32 over a lane's features and a butterfly over the warp's lanes,
// coefficients and sums over support vectors in FP64. The test rows' self dots keep the storage-order FP32 recurrence
// of the other paths (kernelmatrix.cpp:288-296).
#pragma once
#include "common.cuh"

namespace tsvm {

constexpr int FEW_CLASSES = 32;             // the class offsets travel as a kernel argument
constexpr int FEW_TILES = 8;                // row tiles of R rows per call
constexpr int FEW_THREADS = 256, FEW_WARPS = FEW_THREADS / 32;   // one warp more computes the self dots of the test rows
constexpr int FEW_CHUNK = 64;               // support vectors between two barriers
constexpr int FEW_ENTRIES = 2048;           // CSR support vectors: stored entries of all test rows together
constexpr int FEW_SLOTS = 2 * FEW_ENTRIES;  // hash table of their columns

struct FewArgs {
    const float *X;             // dense support vectors, or nullptr
    int ldx;
    const float *val;           // CSR support vectors
    const int *row_ptr, *col;
    int n_sv, d;
    const float *sd_sv;
    const float *T;             // dense test rows, or nullptr
    int dt, ldt;
    const float *tval;          // CSR test rows
    const int *trow_ptr, *tcol;
    int m;
    KernelFn fn;
    const double *coef, *rho;
    int n_classes, n_pairs;
    int start[FEW_CLASSES + 1]; // first support vector of every class, n_sv last
    double *acc;                // [m][n_pairs], zero between calls
    int *ticket;                // [FEW_TILES], zero between calls
    double *dec;                // [m][n_pairs] or nullptr
    int *labels;                // [m] or nullptr
    int *overflow;              // pinned host word: set if the test rows hold more entries than FEW_ENTRIES
};

// Shared memory behind the test rows / the hash table; offsets in bytes from a 16-byte boundary.
template <int R>
struct FewShared {
    static constexpr size_t DOTS = 0;                                              // float [FEW_CHUNK][R]
    static constexpr size_t CLS = DOTS + sizeof(float) * FEW_CHUNK * R;            // int [FEW_CHUNK]
    static constexpr size_t SD = CLS + sizeof(int) * FEW_CHUNK;                    // float [R]
    static constexpr size_t SUMS = (SD + sizeof(float) * R + 15) & ~(size_t) 15;   // double [n_pairs * R]
    static size_t bytes(int n_pairs) { return SUMS + sizeof(double) * n_pairs * R + sizeof(short) * 2 * n_pairs + 16; }
};

// s + sum of x[k]^2 as an FP32 recurrence in storage order; 16 values are in flight ahead of the 16 being added.
__device__ __forceinline__ float self_dot_in_order(const float *x, int n, float s) {
    float now[16], next[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) now[u] = u < n ? x[u] : 0.0f;
    for (int k = 0; k < n; k += 16) {
#pragma unroll
        for (int u = 0; u < 16; ++u) next[u] = k + 16 + u < n ? x[k + 16 + u] : 0.0f;
#pragma unroll
        for (int u = 0; u < 16; ++u) s = fmaf(now[u], now[u], s);
#pragma unroll
        for (int u = 0; u < 16; ++u) now[u] = next[u];
    }
    return s;
}

// One block's share of the support vectors against a tile of R test rows (row_sm, row_ld: dense test rows in shared
// memory). dots_of(s, end, acc): this lane's part of the dot products of support vectors s .. s + 3, those before end.
template <int R, typename Dots>
__device__ __forceinline__ void few_block(const FewArgs &a, const float *row_sm, int row_ld, unsigned char *sm, Dots dots_of) {
    typedef FewShared<R> S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = blockIdx.y * R, rows = a.m - r0 < R ? a.m - r0 : R;
    float *dots = reinterpret_cast<float *>(sm + S::DOTS), *sd_row = reinterpret_cast<float *>(sm + S::SD);
    int *cls = reinterpret_cast<int *>(sm + S::CLS);
    double *sums = reinterpret_cast<double *>(sm + S::SUMS);
    short *pair_i = reinterpret_cast<short *>(sums + a.n_pairs * R), *pair_j = pair_i + a.n_pairs;
    __shared__ bool is_last;
    const int items = a.n_pairs * R;
    for (int e = tid; e < items; e += FEW_THREADS + 32) sums[e] = 0.0;
    for (int i = tid; i < a.n_classes; i += FEW_THREADS + 32)
        for (int j = i + 1; j < a.n_classes; ++j) {
            const int k = i * (2 * a.n_classes - i - 1) / 2 + (j - i - 1);
            pair_i[k] = (short) i; pair_j[k] = (short) j;
        }
    const int per = (a.n_sv + gridDim.x - 1) / gridDim.x;
    const int s0 = blockIdx.x * per, s1 = s0 + per < a.n_sv ? s0 + per : a.n_sv;
    for (int c0 = s0; c0 < s1; c0 += FEW_CHUNK) {
        const int len = s1 - c0 < FEW_CHUNK ? s1 - c0 : FEW_CHUNK;
        if (warp == FEW_WARPS) {
            // self dots of the test rows, in storage order (features beyond d count too); classes of the chunk
            if (c0 == s0 && lane < rows && (a.fn.type == TSVM_RBF || a.fn.type == TSVM_PRECOMPUTED)) {
                if (a.T) {
                    const int known = a.dt < a.d ? a.dt : a.d;      // those are in shared memory already
                    const float s = self_dot_in_order(row_sm + (size_t) lane * row_ld, known, 0.0f);
                    sd_row[lane] = self_dot_in_order(a.T + (size_t) (r0 + lane) * a.ldt + known, a.dt - known, s);
                } else {
                    const int p = a.trow_ptr[r0 + lane];
                    sd_row[lane] = self_dot_in_order(a.tval + p, a.trow_ptr[r0 + lane + 1] - p, 0.0f);
                }
            }
            for (int e = lane; e < len; e += 32) {
                int c = 0;
                while (c + 1 < a.n_classes && c0 + e >= a.start[c + 1]) ++c;
                cls[e] = c;
            }
        } else {
            // four support vectors of a warp at a time: their loads are in flight together
            for (int e = warp * 4; e < len; e += FEW_WARPS * 4) {
                float acc[4][R];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[u][r] = 0.0f;
                dots_of(c0 + e, c0 + len, acc);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        float v = acc[u][r];
                        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                        if (lane == 0 && e + u < len) dots[(e + u) * R + r] = v;
                    }
            }
        }
        __syncthreads();
        for (int e = tid; e < len * R; e += FEW_THREADS + 32) {
            const int r = e % R;
            dots[e] = r < rows ? apply_kernel(a.fn, dots[e], sd_row[r], a.sd_sv[c0 + e / R]) : 0.0f;
        }
        __syncthreads();
        // Decision values: one warp per (row, pair), lanes over the chunk's support vectors
        for (int it = warp; it < items; it += FEW_WARPS + 1) {
            const int r = it % R, k = it / R, i = pair_i[k], j = pair_j[k];
            double s = 0.0;
            for (int e = lane; e < len; e += 32) {
                const int c = cls[e];
                if (c == i) s += a.coef[(size_t) (j - 1) * a.n_sv + c0 + e] * (double) dots[e * R + r];
                else if (c == j) s += a.coef[(size_t) i * a.n_sv + c0 + e] * (double) dots[e * R + r];
            }
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) sums[it] += s;
        }
        __syncthreads();
    }
    for (int it = tid; it < items; it += FEW_THREADS + 32) {
        const int r = it % R, k = it / R;
        if (r < rows && sums[it] != 0.0) atomicAdd(a.acc + (size_t) (r0 + r) * a.n_pairs + k, sums[it]);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) is_last = atomicAdd(a.ticket + blockIdx.y, 1) == (int) gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int it = tid; it < items; it += FEW_THREADS + 32) {
        const int r = it % R, k = it / R;
        if (r >= rows) continue;
        const size_t at = (size_t) (r0 + r) * a.n_pairs + k;
        const double v = __ldcg(a.acc + at) - a.rho[k];
        a.acc[at] = 0.0;
        if (a.dec) a.dec[at] = v;
        sums[it] = v;
    }
    if (tid == 0) a.ticket[blockIdx.y] = 0;
    if (!a.labels) return;
    __syncthreads();
    // votes -> index of the winning class, first maximum wins: one warp per row, one lane per class
    for (int r = warp; r < rows; r += FEW_WARPS + 1) {
        int votes = 0;
        for (int k = 0; k < a.n_pairs; ++k) {
            const bool pos = sums[k * R + r] > 0;
            if ((pos && pair_i[k] == lane) || (!pos && pair_j[k] == lane)) ++votes;
        }
        const int key = lane < a.n_classes ? votes * 64 + (63 - lane) : -1;
        const int best = __reduce_max_sync(0xffffffffu, key);
        if (lane == 0) a.labels[r0 + r] = 63 - (best & 63);
    }
}

// Dense support vectors: lanes over groups of four features, the test rows (zero padded) in shared memory.
template <int R>
__global__ void __launch_bounds__(FEW_THREADS + 32) predict_few_dense_kernel(const FewArgs a) {
    extern __shared__ __align__(16) unsigned char few_sm[];
    const int dp = (a.d + 3) & ~3, tid = threadIdx.x, lane = tid & 31;
    float *rows_sm = reinterpret_cast<float *>(few_sm);                 // [R][dp]
    const int r0 = blockIdx.y * R;
    if (a.T) {
        const int lim = a.dt < a.d ? a.dt : a.d;
        for (int e = tid; e < R * dp; e += FEW_THREADS + 32) {
            const int r = e / dp, k = e - r * dp;
            rows_sm[e] = r0 + r < a.m && k < lim ? a.T[(size_t) (r0 + r) * a.ldt + k] : 0.0f;
        }
    } else {
        for (int e = tid; e < R * dp; e += FEW_THREADS + 32) rows_sm[e] = 0.0f;
        __syncthreads();
        for (int r = 0; r < R && r0 + r < a.m; ++r)
            for (int p = a.trow_ptr[r0 + r] + tid; p < a.trow_ptr[r0 + r + 1]; p += FEW_THREADS + 32)
                if (a.tcol[p] < a.d) rows_sm[r * dp + a.tcol[p]] = a.tval[p];
    }
    __syncthreads();
    few_block<R>(a, rows_sm, dp, few_sm + sizeof(float) * (size_t) R * dp, [&](int s, int end, float (&acc)[4][R]) {
        const float4 *x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = reinterpret_cast<const float4 *>(a.X + (size_t) (s + u < end ? s + u : end - 1) * a.ldx);
        for (int k = lane; k < dp / 4; k += 32) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = __ldg(x[u] + k);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float4 t = reinterpret_cast<const float4 *>(rows_sm + (size_t) r * dp)[k];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    acc[u][r] = fmaf(v[u].w, t.w, fmaf(v[u].z, t.z, fmaf(v[u].y, t.y, fmaf(v[u].x, t.x, acc[u][r]))));
            }
        }
    });
}

// CSR support vectors against CSR test rows: lanes over a support vector's stored entries; the columns of the test
// rows are in a hash table, so an entry whose column no test row has - nearly all of them for text - costs one probe.
template <int R>
__global__ void __launch_bounds__(FEW_THREADS + 32) predict_few_csr_kernel(const FewArgs a) {
    extern __shared__ __align__(16) unsigned char few_sm[];
    float *values = reinterpret_cast<float *>(few_sm);                          // [FEW_ENTRIES][R]
    int *key = reinterpret_cast<int *>(values + FEW_ENTRIES * R);               // [FEW_SLOTS]
    short *entry = reinterpret_cast<short *>(key + FEW_SLOTS);                  // [FEW_SLOTS]
    __shared__ int n_entries;
    const int tid = threadIdx.x, lane = tid & 31, r0 = blockIdx.y * R, r1 = r0 + R < a.m ? r0 + R : a.m;
    auto home = [](int c) { return (unsigned) (c * 2654435761u) >> 20; };       // 12 bits
    static_assert(FEW_SLOTS == 4096, "home() yields 12 bits");
    for (int e = tid; e < FEW_SLOTS; e += FEW_THREADS + 32) key[e] = -1;
    if (tid == 0) n_entries = 0;
    __syncthreads();
    const int p0 = a.trow_ptr[r0], p1 = a.trow_ptr[r1];
    if (p1 - p0 > FEW_ENTRIES) {                // the caller's count was wrong: it falls back to the general path
        if (tid == 0) *a.overflow = 1;
        return;
    }
    for (int p = p0 + tid; p < p1; p += FEW_THREADS + 32) {
        const int c = a.tcol[p];
        if (c >= a.d) continue;
        for (unsigned s = home(c);; s = (s + 1) & (FEW_SLOTS - 1)) {
            const int old = atomicCAS(&key[s], -1, c);
            if (old == -1) {
                const int e = atomicAdd(&n_entries, 1);
                entry[s] = (short) e;
#pragma unroll
                for (int r = 0; r < R; ++r) values[e * R + r] = 0.0f;
                break;
            }
            if (old == c) break;
        }
    }
    __syncthreads();
    auto find = [&](int c) -> int {
        for (unsigned s = home(c);; s = (s + 1) & (FEW_SLOTS - 1)) {
            const int k = key[s];
            if (k == c) return entry[s];
            if (k == -1) return -1;
        }
    };
    for (int r = r0; r < r1; ++r)
        for (int p = a.trow_ptr[r] + tid; p < a.trow_ptr[r + 1]; p += FEW_THREADS + 32)
            if (a.tcol[p] < a.d) values[find(a.tcol[p]) * R + (r - r0)] = a.tval[p];
    __syncthreads();
    constexpr size_t table = sizeof(float) * FEW_ENTRIES * R + (sizeof(int) + sizeof(short)) * FEW_SLOTS;
    static_assert(table % 16 == 0, "what follows the table is 16-byte aligned");
    few_block<R>(a, nullptr, 0, few_sm + table, [&](int s, int end, float (&acc)[4][R]) {
        int p[4], e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            p[u] = s + u < end ? a.row_ptr[s + u] + lane : 0;
            e[u] = s + u < end ? a.row_ptr[s + u + 1] : 0;
        }
        bool more = true;
        while (more) {
            int c[4];
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                c[u] = p[u] < e[u] ? a.col[p[u]] : -2;
                v[u] = p[u] < e[u] ? a.val[p[u]] : 0.0f;
                p[u] += 32;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int at = c[u] >= 0 ? find(c[u]) : -1;
                if (at >= 0) {
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[u][r] = fmaf(v[u], values[at * R + r], acc[u][r]);
                }
            }
            more = p[0] < e[0] || p[1] < e[1] || p[2] < e[2] || p[3] < e[3];
        }
    });
}

}  // namespace tsvm
