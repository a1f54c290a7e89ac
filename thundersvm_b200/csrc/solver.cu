// Batched SMO solver on the device: working-set selection (radix top-k over (f, id) keys),
// the one-CTA local solver, the fused f update and the outer loop with the reference's
// termination rules. Reference behaviour: src/thundersvm/solver/csmosolver.cpp:10-239,
// src/thundersvm/solver/nusmosolver.cpp:9-136, src/thundersvm/kernel/smo_kernel.cu:28-315.
#include "common.cuh"
#include "local_smo.cuh"
#include "select.cuh"
#include <chrono>
#include <limits.h>
#include <string.h>
#include <stdlib.h>
#include <sched.h>
#include <dlfcn.h>
#include <mutex>
#include <vector>

namespace tsvm {

// ---- gather of the working set's block and vectors ---------------------------------------------
// Logical slot t of the working set lives in physical row phys(t) of the row buffer (the two
// halves of the buffer swap roles every outer iteration instead of being copied).
__device__ __forceinline__ int phys_row(int t, int q, int first_half_phys) {
    return t < q ? first_half_phys * q + t : (1 - first_half_phys) * q + (t - q);
}

constexpr int GATHER_AT_A_TIME = 4;
__global__ void gather_ws_kernel(int ws, int q, int first_half_phys, const int *__restrict__ ids,
                                 const float *__restrict__ rows, long long ld, const float *__restrict__ diag,
                                 const int *__restrict__ y, const double *__restrict__ f,
                                 const double *__restrict__ alpha, float *__restrict__ kww,
                                 float *__restrict__ diag_ws, int *__restrict__ y_ws, double *__restrict__ f_ws,
                                 double *__restrict__ alpha_ws, int block_rows, const int *__restrict__ row_slot,
                                 PhaseTimes *times) {
    const int a = blockIdx.x;                      // logical slot of the row
    if (times && a == 0 && threadIdx.x == 0) times->rows_end = device_ns();
    // rows >= block_rows of the block are written by someone else (the overlapped iteration computes them
    // directly); the slot vectors are gathered for every slot
    // a slot without an instance (id -1: fewer eligible instances than slots) is inert: y = 0 puts it in no set
    if (a < block_rows) {
        const float *row = rows + (size_t) (row_slot ? row_slot[a] : phys_row(a, q, first_half_phys)) * ld;
        // all of a thread's ids first, then all of its values: two latencies instead of eight
        for (int b0 = threadIdx.x; b0 < ws; b0 += GATHER_AT_A_TIME * blockDim.x) {
            int id[GATHER_AT_A_TIME];
            float k[GATHER_AT_A_TIME];
#pragma unroll
            for (int u = 0; u < GATHER_AT_A_TIME; ++u) id[u] = b0 + u * blockDim.x < ws ? ids[b0 + u * blockDim.x] : -1;
#pragma unroll
            for (int u = 0; u < GATHER_AT_A_TIME; ++u) k[u] = id[u] >= 0 ? row[id[u]] : 0.0f;
#pragma unroll
            for (int u = 0; u < GATHER_AT_A_TIME; ++u)
                if (b0 + u * blockDim.x < ws) kww[(size_t) a * ws + b0 + u * blockDim.x] = k[u];
        }
    }
    if (threadIdx.x == 0) {
        const int id = ids[a];
        if (id >= 0) { diag_ws[a] = diag[id]; y_ws[a] = y[id]; f_ws[a] = f[id]; alpha_ws[a] = alpha[id]; }
        else { diag_ws[a] = 1.0f; y_ws[a] = 0; f_ws[a] = 0.0; alpha_ws[a] = 0.0; }
    }
}

// =================================================================================================
// Kernel-row cache: least-recently-used rows kept in HBM
// =================================================================================================
// The reference keeps only the previous iteration's q rows (csmosolver.cpp:69,75). Here the row buffer has
// room for `cap` rows (as many as the memory budget allows, at least ws + q). A directory on the device maps
// instance -> row (slot_of), row -> instance (inst_of) and row -> outer iteration of its last use (stamp).
// After every selection one block looks the new members up: a hit only points the member's slot at the cached
// row; the misses are compacted into the list the kernel-row engine then computes, and each gets the row of a
// victim - the rows with the oldest stamps that do not belong to the current working set, found with a
// histogram over the stamps; ties go to the lower row number, so the choice does not depend on thread timing.
// Everything stays on the device: the engine reads the number of misses from memory.
constexpr int CACHE_THREADS = 1024, CACHE_BINS = 2048;
enum { CACHE_N_MISS = 0, CACHE_HITS = 1, CACHE_MISSES = 2, CACHE_BLOCKS = 3, CACHE_BLOCKS_SAVED = 4,
       CACHE_NEXT_FREE = 5,         // rows [0, next_free) have been handed out; the rest never held a row
       CACHE_CTRS = 8 };

__device__ __forceinline__ int cache_bin(int stamp, int now) {
    // older -> smaller bin; never-used rows (stamp 0) are the oldest; rows used in this iteration are not candidates
    if (stamp <= 0) return 0;
    const int age = now - stamp;
    return age >= CACHE_BINS - 1 ? 0 : CACHE_BINS - 1 - age;
}

__global__ void __launch_bounds__(CACHE_THREADS, 1)
cache_assign_kernel(const int *__restrict__ ids, int t0, int n_new, int now, int *__restrict__ slot_of,
                    int *__restrict__ inst_of, int *__restrict__ stamp, int cap,
                    const int *__restrict__ row_slot_before, int *__restrict__ row_slot,
                    int *__restrict__ miss_ids, int *__restrict__ miss_slot, int *__restrict__ victims,
                    long long *__restrict__ ctr, int row_block, const int *__restrict__ stop, PhaseTimes *times) {
    if (stop && *stop) {            // queued past the end of a solve: no member changes, no row to compute
        if (threadIdx.x == 0) reinterpret_cast<int *>(ctr)[0] = 0;
        return;
    }
    __shared__ int hist[CACHE_BINS];
    __shared__ int miss_t[CACHE_THREADS];
    __shared__ int wsum[32], wpre_b[32], wpre_sel[32];
    __shared__ int n_miss_s, thr_bin, need_s, n_hit_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the members that stay move to the front; their rows are in use now
    int keep = 0;
    if (tid < t0) keep = row_slot_before[t0 + tid];
    for (int b = tid; b < CACHE_BINS; b += CACHE_THREADS) hist[b] = 0;
    if (tid == 0) { n_miss_s = 0; n_hit_s = 0; }
    __syncthreads();
    if (tid < t0) { row_slot[tid] = keep; if (ids[tid] >= 0) stamp[keep] = now; }
    // look the new members up; misses are compacted in member order
    int id = -1, s = -1;
    if (tid < n_new) {
        id = ids[t0 + tid];
        s = id >= 0 ? slot_of[id] : -1;
        if (id < 0) row_slot[t0 + tid] = 0;            // an empty working-set slot is inert: any row will do
        else if (s >= 0) { row_slot[t0 + tid] = s; stamp[s] = now; }
    }
    const bool miss = tid < n_new && id >= 0 && s < 0;
    const unsigned mb = __ballot_sync(0xffffffffu, miss);
    if (lane == 0) wsum[warp] = __popc(mb);
    const unsigned hb = __ballot_sync(0xffffffffu, tid < n_new && id >= 0 && s >= 0);
    if (lane == 0 && hb) atomicAdd(&n_hit_s, __popc(hb));
    __syncthreads();
    if (warp == 0) {
        const int v = wsum[lane];
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int a = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += a; }
        wsum[lane] = inc - v;
        if (lane == 31) n_miss_s = inc;
    }
    __syncthreads();
    if (miss) miss_t[wsum[warp] + __popc(mb & ((1u << lane) - 1))] = tid;
    const int n_miss = n_miss_s;
    // (the stamps written above must be visible to the sweeps below)
    __threadfence_block();
    __syncthreads();
    // While rows that never held anything are left, the misses take the lowest of them - the rows the sweeps
    // below would pick (stamp 0 is the oldest, ties go to the lower row) without sweeping the stamps.
    __shared__ long long next_free_s;
    if (tid == 0) next_free_s = ctr[CACHE_NEXT_FREE];
    __syncthreads();
    const long long next_free = next_free_s;
    const bool fresh = next_free + n_miss <= cap;
    if (n_miss > 0 && fresh) {
        if (tid < n_miss) victims[tid] = (int) next_free + tid;
        __threadfence_block();
        __syncthreads();
    } else if (n_miss > 0) {
        // histogram of the candidates' stamps
        for (int r = tid; r < cap; r += CACHE_THREADS) {
            const int st = stamp[r];
            if (st != now) atomicAdd(&hist[cache_bin(st, now)], 1);
        }
        __syncthreads();
        // threshold bin: the n_miss oldest rows are all rows of the bins below it and `need` rows of the bin itself
        if (warp == 0) {
            int run = 0, found = 0;
            for (int b0 = 0; b0 < CACHE_BINS && !found; b0 += 32) {
                const int v = hist[b0 + lane];
                int inc = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const int a = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += a; }
                const unsigned reach = __ballot_sync(0xffffffffu, run + inc >= n_miss);
                if (reach) {
                    const int l = __ffs(reach) - 1;
                    const int before = run + __shfl_sync(0xffffffffu, inc - v, l);
                    if (lane == 0) { thr_bin = b0 + l; need_s = n_miss - before; }
                    found = 1;
                }
                run += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (!found && lane == 0) { thr_bin = CACHE_BINS; need_s = 0; }     // cannot happen: cap >= ws + q
        }
        __syncthreads();
        const int B = thr_bin, need = need_s;
        // ordered choice: every warp owns a contiguous range of rows
        const int per = (cap + 31) / 32;
        const int r0 = warp * per, r1 = min(cap, r0 + per);
        int cnt_b = 0, cnt_l = 0;
        for (int r = r0 + lane; r - lane < r1; r += 32) {
            const int st = r < r1 ? stamp[r] : now;
            const int bin = st != now ? cache_bin(st, now) : CACHE_BINS;
            cnt_b += __popc(__ballot_sync(0xffffffffu, bin == B));
            cnt_l += __popc(__ballot_sync(0xffffffffu, bin < B));
        }
        if (lane == 0) { wpre_b[warp] = cnt_b; wpre_sel[warp] = cnt_l; }
        __syncthreads();
        if (warp == 0) {
            const int vb = wpre_b[lane], vl = wpre_sel[lane];
            int ib = vb;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int a = __shfl_up_sync(0xffffffffu, ib, o); if (lane >= o) ib += a; }
            const int pre_b = ib - vb;
            const int take_b = max(0, min(vb, need - pre_b));
            int isel = vl + take_b;
            const int vsel = isel;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int a = __shfl_up_sync(0xffffffffu, isel, o); if (lane >= o) isel += a; }
            wpre_b[lane] = pre_b;
            wpre_sel[lane] = isel - vsel;
        }
        __syncthreads();
        int run_b = wpre_b[warp], pos = wpre_sel[warp];
        for (int r = r0 + lane; r - lane < r1; r += 32) {
            const int st = r < r1 ? stamp[r] : now;
            const int bin = st != now ? cache_bin(st, now) : CACHE_BINS;
            const unsigned bb = __ballot_sync(0xffffffffu, bin == B);
            const int rank_b = run_b + __popc(bb & ((1u << lane) - 1));
            const bool sel = bin < B || (bin == B && rank_b < need);
            const unsigned sb = __ballot_sync(0xffffffffu, sel);
            if (sel) victims[pos + __popc(sb & ((1u << lane) - 1))] = r;
            run_b += __popc(bb);
            pos += __popc(sb);
        }
        __threadfence_block();
        __syncthreads();
    }
    if (n_miss > 0) {
        // the misses take the victims' rows
        if (tid < n_miss) {
            const int t = miss_t[tid];
            const int mid = ids[t0 + t];
            const int r = victims[tid];
            const int old = inst_of[r];
            if (old >= 0) slot_of[old] = -1;
            inst_of[r] = mid;
            slot_of[mid] = r;
            stamp[r] = now;
            row_slot[t0 + t] = r;
            miss_ids[tid] = mid;
            miss_slot[tid] = r;
        }
    }
    if (tid == 0) {
        times->select_end = device_ns();
        reinterpret_cast<int *>(ctr)[0] = n_miss;                 // CACHE_N_MISS, read by the engines as an int
        ctr[CACHE_HITS] += n_hit_s;
        ctr[CACHE_MISSES] += n_miss;
        ctr[CACHE_BLOCKS] += (n_new + row_block - 1) / row_block;
        ctr[CACHE_BLOCKS_SAVED] += (n_new + row_block - 1) / row_block - (n_miss + row_block - 1) / row_block;
        ctr[CACHE_NEXT_FREE] = fresh ? next_free + n_miss : (long long) cap;
    }
}

// ---- end-of-iteration bookkeeping on the device ----------------------------------------------------
// The reference decides after every outer iteration, on the host, whether to go on (csmosolver.cpp:83-111).
// Here one thread applies the same rules to the same doubles on the device, so the host can queue several
// iterations and read the outcome once: every kernel of a queued iteration looks at `stop` first and does
// nothing once it is set.
struct SolverState {
    int stop;                       // first member: kernels take a pointer to it
    int done;                       // the reference's own termination rules fired
    int iter, same_cnt, swap_cnt;
    int short_got, short_wanted;    // a selection that could not fill its slots (got < wanted)
    int engine_status;              // non-zero: a bounded wait of the kernel-row engine ran out
    double prev, last, second_last, diff0;
    long long local_iter;
    long long ctr[CACHE_CTRS];      // cache counters as of the last iteration that ran
    PhaseTimes times;               // of the running iteration
    long long update_begin;         // of the iteration before
    long long ns_select, ns_rows, ns_local, ns_update;     // sums over the iterations that ran
};
static_assert(offsetof(SolverState, stop) == 0, "kernels read the stop flag through a pointer to the struct");
// Next to it when the blocks of an iteration's f update left, by the iteration's parity: written while the block that ends the
// iteration writes the state back, read by the iteration after.
struct SolverCtl : SolverState {
    long long update_end[2];
};

struct StatusArgs {
    SolverCtl *c = nullptr;         // nullptr: nothing to do
    const double *diff = nullptr;
    const int *got = nullptr;
    int wanted = 0;
    double eps = 0;
    int max_iter = -1;
    const long long *cache_ctr = nullptr;
    const int *engine_status = nullptr;
    int *ids = nullptr;
    int q = 0;
    unsigned char *in_ws = nullptr;
    volatile unsigned long long *progress = nullptr;
    int parity = 0;                 // of the iteration
};

// One block. It reads nothing that the f update writes, so that it runs as one more block of the iteration's last f update
// (a launch of its own took 4.1 us and 2.2 between launches).
__device__ __noinline__ void solver_status(const StatusArgs &s) {
    SolverCtl *c = s.c;
    const long long begin = device_ns();        // of the f update that this block runs in: its other blocks start with it
    const int already = c->stop;
    __syncthreads();
    if (already) return;
    // The working set rotates for the next selection: the old second half becomes the first half and keeps its flags,
    // the old first half leaves. (After the last iteration nothing looks at it again.)
    for (int t = threadIdx.x; t < s.q; t += blockDim.x) {
        const int leaving = s.ids[t], staying = s.ids[s.q + t];
        if (leaving >= 0) s.in_ws[leaving] = 0;
        if (staying >= 0) s.in_ws[staying] = 1;
        s.ids[t] = staying;
    }
    if (threadIdx.x != 0) return;
    // everything is read before anything is written, so that the reads are in flight together (5.2 -> 4.4 us against
    // reads that each waited for the write before them)
    SolverState v = *c;
    const long long update_end = *(volatile const long long *) &c->update_end[s.parity ^ 1];       // (of the iteration before)
    const double d = s.diff[0], steps = s.diff[1], eps = s.eps;
    const int found = *s.got, engine = s.engine_status ? *s.engine_status : 0;
    if (s.cache_ctr)
#pragma unroll
        for (int k = 0; k < CACHE_CTRS; ++k) v.ctr[k] = s.cache_ctr[k];
    v.diff0 = d;
    v.local_iter += (long long) steps;
    // csmosolver.cpp:86-111
    if (fabs(d - v.prev) < eps * 0.001) v.same_cnt++;
    else { v.same_cnt = 0; v.prev = d; }
    if (fabs(d - v.second_last) < eps * 0.001) v.swap_cnt++;
    else v.swap_cnt = 0;
    v.second_last = v.last;
    v.last = d;
    if ((v.same_cnt >= 10 && fabs(d - 2.0) > eps) || d < eps || (v.swap_cnt >= 10 && fabs(d - 2.0) > eps)) v.stop = v.done = 1;
    v.iter++;
    if (s.max_iter != -1 && v.iter - 1 == s.max_iter) v.stop = 1;     // iteration cap (csmosolver.cpp:110)
    if (found < s.wanted) { v.short_got = found; v.short_wanted = s.wanted; v.stop = 1; }
    if (engine) { v.engine_status = engine; v.stop = 1; }
    if (s.progress) {
        // how far the solve is, for the host that waits for it: a word of pinned host memory
        *s.progress = ((unsigned long long) v.iter << 1) | (unsigned) v.stop;
        v.ns_select += v.times.select_end - v.times.select_begin;
        v.ns_rows += v.times.rows_end - v.times.select_end;
        v.ns_local += v.times.local_end - v.times.local_begin;
        if (update_end > v.update_begin && v.update_begin) v.ns_update += update_end - v.update_begin;
        v.update_begin = begin;
    }
    *static_cast<SolverState *>(c) = v;
}

__global__ void solver_status_kernel(const StatusArgs s) { solver_status(s); }

// *any becomes non-zero if one of a[0..n) is
__global__ void any_nonzero_kernel(const double *__restrict__ a, int n, int *__restrict__ any) {
    bool mine = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) mine = mine || a[i] != 0.0;
    if (__syncthreads_or(mine) && threadIdx.x == 0) *any = 1;
}

__global__ void fill_int_kernel(int *p, long long n, int v) {
    for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) p[i] = v;
}

// =================================================================================================
// f update:  f[j] -= sum_t alpha_diff[t] * rows[phys(t)][j]   (smo_kernel.cu:289-310)
// =================================================================================================
// What bounds it: HBM for many columns (a row is read once, 4 bytes per column), the latency of the reads for few. The rows
// with a non-zero alpha_diff are therefore split into eight runs, one per warp of a block, 16 (V = 1) or 8 (V = 4) rows in
// flight per lane; the runs' sums are added in order. The split depends on the number of rows alone, so that a column's
// sum has the same bits for any number of columns, V and share of them on this GPU. Measured, 512 rows, against one thread
// per column (four from 300,000 on): 1,000 columns 41 -> 10 us, 10,000 39 -> 12, 32,768 42 -> 20, 100,000 53 -> 45, 200,000
// 100 -> 78 (5.3 TB/s), 400,000 140 -> 141.
// Slots [t_begin, t_mid) and [t_mid, t_end) are two sums, subtracted one after the other as two launches would do (one
// launch for both halves of a working set: 3.9 us less per iteration).
constexpr int UPD_WARPS = 8, UPD_SLOTS = 1024;
constexpr int UPD_WIDE_PER_SM = 2, UPD_NARROW_PER_SM = 3;        // blocks of the V = 4 form and of the others that fit an SM (registers)
template <int V>
__global__ void __launch_bounds__(UPD_WARPS * 32, V == 4 ? UPD_WIDE_PER_SM : UPD_NARROW_PER_SM)
update_f_kernel(double *__restrict__ f, int n, const double *__restrict__ alpha_diff, int q, int first_half_phys,
                const float *__restrict__ rows, long long ld, int t_begin, int t_mid, int t_end, const int *__restrict__ row_slot,
                const StatusArgs status) {
    const int other = status.c != nullptr, blocks = gridDim.x - other, block = blockIdx.x - other;
    if (block < 0) { solver_status(status); return; }               // the first block ends the iteration instead
    constexpr int U = V == 4 ? 8 : 16;
    __shared__ double ad[UPD_SLOTS], part[2][UPD_WARPS][32 * V];
    __shared__ int prow[UPD_SLOTS], count[UPD_WARPS], count_first[UPD_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // order-preserving compaction of the non-zero entries of slots [t_begin, t_end): 128 slots per warp
    constexpr int PER = UPD_SLOTS / UPD_WARPS / 32;
    double dv[PER];
    int pr[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int t = t_begin + (warp * PER + k) * 32 + lane;
        dv[k] = t < t_end ? alpha_diff[t] : 0.0;
        pr[k] = t < t_end ? (row_slot ? row_slot[t] : (q > 0 ? phys_row(t, q, first_half_phys) : t)) : 0;
    }
    int mine = 0, mine_first = 0;
    unsigned ballot[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        ballot[k] = __ballot_sync(0xffffffffu, dv[k] != 0.0);
        mine += __popc(ballot[k]);
        mine_first += __popc(__ballot_sync(0xffffffffu, dv[k] != 0.0 && t_begin + (warp * PER + k) * 32 + lane < t_mid));
    }
    if (lane == 0) { count[warp] = mine; count_first[warp] = mine_first; }
    __syncthreads();
    int base = 0, m = 0, m_first = 0;
#pragma unroll
    for (int w = 0; w < UPD_WARPS; ++w) {
        if (w < warp) base += count[w];
        m += count[w];
        m_first += count_first[w];
    }
    if (m == 0) return;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        if (dv[k] != 0.0) {
            const int p = base + __popc(ballot[k] & ((1u << lane) - 1));
            ad[p] = dv[k];
            prow[p] = pr[k];
        }
        base += __popc(ballot[k]);
    }
    __syncthreads();
    int buf = 0;
    for (long long c0 = (long long) block * (32 * V); c0 < n;) {
        double f_now = tid < 32 * V && c0 + tid < n ? f[c0 + tid] : 0.0;
        const float *col = rows + (c0 + lane * V < n ? c0 + lane * V : 0);
        auto load = [&](int r, float (&x)[V]) {
            const float *at = col + (size_t) prow[r] * ld;
            if constexpr (V == 2) {
                const float2 t = __ldcs(reinterpret_cast<const float2 *>(at));
                x[0] = t.x; x[1] = t.y;
            } else if constexpr (V == 4) {
                const float4 t = __ldcs(reinterpret_cast<const float4 *>(at));       // (the row is padded to a multiple of 4)
                x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
            } else x[0] = __ldcs(at);
        };
        for (int part_no = 0; part_no < 2; ++part_no) {         // the slots before t_mid, then those from there on
            const int p0 = part_no ? m_first : 0, p1 = part_no ? m : m_first;
            if (p0 == p1) continue;
            const int run = (p1 - p0 + UPD_WARPS - 1) / UPD_WARPS, r0 = p0 + warp * run, r1 = min(p1, r0 + run);
            double s[V];
#pragma unroll
            for (int v = 0; v < V; ++v) s[v] = 0;
            for (int r = r0; r < r1; r += U) {
                float x[U][V];
                if (r + U <= r1) {
#pragma unroll
                    for (int u = 0; u < U; ++u) load(r + u, x[u]);
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int v = 0; v < V; ++v) s[v] += ad[r + u] * x[u][v];
                } else {                            // the rest in one go as well
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (r + u < r1) load(r + u, x[u]);
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (r + u < r1)
#pragma unroll
                            for (int v = 0; v < V; ++v) s[v] += ad[r + u] * x[u][v];
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v) part[buf][warp][lane * V + v] = s[v];
            __syncthreads();        // (this buffer is written again only after the next barrier)
            if (tid < 32 * V && c0 + tid < n) {
                double t = part[buf][0][tid];
#pragma unroll
                for (int w = 1; w < UPD_WARPS; ++w) t += part[buf][w][tid];
                f_now -= t;
            }
            buf ^= 1;
        }
        if (tid < 32 * V && c0 + tid < n) f[c0 + tid] = f_now;
        if (V < 4) break;                       // one tile per block
        c0 += (long long) blocks * (32 * V);
    }
    if (status.c && tid == 0)
        atomicMax(reinterpret_cast<unsigned long long *>(&status.c->update_end[status.parity]), (unsigned long long) device_ns());
}

// =================================================================================================
// rho / objective
// =================================================================================================
// out[0..12] = n_free(+), sum_free f(+), n_free(-), sum_free f(-), sum of the objective terms,
//              min f over I_up (+), max f over I_low (+), the same two for (-),
//              max f over I_up (+), min f over I_low (+), the same two for (-).
constexpr int RHO_VALS = 13;
__global__ void __launch_bounds__(1024)
rho_obj_kernel(int n, const double *__restrict__ f, const double *__restrict__ alpha, const int *__restrict__ y,
               double Cp, double Cn, double *__restrict__ out) {
    __shared__ double sh[32][RHO_VALS];
    double v[RHO_VALS] = {0, 0, 0, 0, 0, INFINITY, -INFINITY, INFINITY, -INFINITY, -INFINITY, INFINITY, -INFINITY,
                          INFINITY};
    for (int i = threadIdx.x; i < n; i += 1024) {
        const double a = alpha[i], fi = f[i];
        const int yi = y[i];
        v[4] += a - (fi + yi) * a * yi / 2;
        const bool up = in_I_up(a, yi, Cp, Cn), low = in_I_low(a, yi, Cp, Cn);
        if (yi > 0) {
            if (a > 0 && a < Cp) { v[0] += 1; v[1] += fi; }
            if (up) { v[5] = fmin(v[5], fi); v[9] = fmax(v[9], fi); }
            if (low) { v[6] = fmax(v[6], fi); v[10] = fmin(v[10], fi); }
        } else {
            if (a > 0 && a < Cn) { v[2] += 1; v[3] += fi; }
            if (up) { v[7] = fmin(v[7], fi); v[11] = fmax(v[11], fi); }
            if (low) { v[8] = fmax(v[8], fi); v[12] = fmin(v[12], fi); }
        }
    }
    auto combine = [](int k, double a, double b) -> double {
        if (k < 5) return a + b;
        const bool is_min = (k == 5 || k == 7 || k == 10 || k == 12);
        return is_min ? fmin(a, b) : fmax(a, b);
    };
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int k = 0; k < RHO_VALS; ++k) v[k] = combine(k, v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < RHO_VALS; ++k) sh[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w)
            for (int k = 0; k < RHO_VALS; ++k) sh[0][k] = combine(k, sh[0][k], sh[w][k]);
        for (int k = 0; k < RHO_VALS; ++k) out[k] = sh[0][k];
    }
}

__global__ void scale_kernel(double *a, int n, double r) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] /= r;
}

// =================================================================================================
// Column-sharded solver: per-rank device work of one outer iteration (the exchange steps between the
// phases belong to the caller)
// =================================================================================================

// all-gathered candidate lists [world][lists][want] -> [lists][world * want]
__global__ void shard_regroup_kernel(const double *__restrict__ gf, const int *__restrict__ gi, int world, int lists,
                                     int want, double *__restrict__ of, int *__restrict__ oi) {
    const int total = world * lists * want;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int r = e / (lists * want), rem = e - r * lists * want, l = rem / want, p = rem - l * want;
        const size_t o = (size_t) l * world * want + (size_t) r * want + p;
        of[o] = gf[e];
        oi[o] = gi[e];
    }
}

// Slots 0..q-1 <- slots q..ws-1 (global ids and per-member vectors); in-working-set flags of the owned
// instances: the old first half leaves, the old second half stays. One block, q <= 512.
__global__ void shard_shift_kernel(int *ids, int q, int lo, int hi, unsigned char *in_ws, float *m_sd,
                                   float *m_unscale, float *m_diag) {
    const int t = threadIdx.x;
    if (t < q) {
        const int leaving = ids[t], staying = ids[q + t];
        if (leaving >= lo && leaving < hi) in_ws[leaving - lo] = 0;
        if (staying >= lo && staying < hi) in_ws[staying - lo] = 1;
        ids[t] = staying;
        m_sd[t] = m_sd[q + t]; m_unscale[t] = m_unscale[q + t]; m_diag[t] = m_diag[q + t];
    }
}

// What this rank contributes to the exchange after the selection: for the n_new new members (slots slot0..)
// their feature row, self dot and diagonal (zeros if another rank owns them) -> crow[s][0..d), [dp], [dp+1]
// (row stride ldw = dp + 4, dp = round_up(d, 4)); for all ws members (y, f, alpha) -> cstate[slot][3].
// Summing the contributions of all ranks gives the values (adding zeros is exact).
__global__ void shard_contrib_kernel(const int *__restrict__ ids, int slot0, int n_new, int ws, int lo, int hi,
                                     const float *__restrict__ X, int ldx, int d, int dp, const float *__restrict__ sd,
                                     const float *__restrict__ diag, const int *__restrict__ y,
                                     const double *__restrict__ f, const double *__restrict__ alpha,
                                     float *__restrict__ crow, double *__restrict__ cstate) {
    const int b = blockIdx.x;
    if (b < n_new) {
        const int gid = ids[slot0 + b];
        const bool own = gid >= lo && gid < hi;
        float *dst = crow + (size_t) b * (dp + 4);
        const float *src = own ? X + (size_t) (gid - lo) * ldx : nullptr;
        for (int k = threadIdx.x; k < dp + 4; k += blockDim.x) {
            float v = 0.0f;
            if (own) {
                if (k < d) v = src[k];
                else if (k == dp) v = sd[gid - lo];
                else if (k == dp + 1) v = diag[gid - lo];
            }
            dst[k] = v;
        }
    } else {
        for (int t = (b - n_new) * blockDim.x + threadIdx.x; t < ws; t += (gridDim.x - n_new) * blockDim.x) {
            const int gid = ids[t];
            const bool own = gid >= lo && gid < hi;
            cstate[3 * t] = own ? (double) y[gid - lo] : 0.0;
            cstate[3 * t + 1] = own ? f[gid - lo] : 0.0;
            cstate[3 * t + 2] = own ? alpha[gid - lo] : 0.0;
        }
    }
}

// After the exchange: member vectors of the new slots out of the row buffer, solver inputs out of the state.
__global__ void shard_unpack_kernel(const float *__restrict__ crow, int slot0, int n_new, int dp, int ws,
                                    const double *__restrict__ cstate, float *__restrict__ m_sd,
                                    float *__restrict__ m_diag, int *__restrict__ y_ws, double *__restrict__ f_ws,
                                    double *__restrict__ a_ws) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_new) {
        m_sd[slot0 + t] = crow[(size_t) t * (dp + 4) + dp];
        m_diag[slot0 + t] = crow[(size_t) t * (dp + 4) + dp + 1];
    }
    if (t < ws) {
        y_ws[t] = (int) cstate[3 * t];
        f_ws[t] = cstate[3 * t + 1];
        a_ws[t] = cstate[3 * t + 2];
    }
}

// alpha of the owned members back into the rank's slice
__global__ void shard_scatter_kernel(const int *__restrict__ ids, int ws, int lo, int hi,
                                     const double *__restrict__ a_ws, double *__restrict__ alpha) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ws) {
        const int gid = ids[t];
        if (gid >= lo && gid < hi) alpha[gid - lo] = a_ws[t];
    }
}

// =================================================================================================
// host side
// =================================================================================================
// f -= the rows of slots [t0, t1) times their alpha_diff, those before t_mid first. 16-byte loads, 128 columns at a time by blocks
// that stay (a tile's reads start while the last one is being added up), where these tiles keep one and a half blocks per SM
// busy: 20 against 23 us at 32,768 columns, but 18.5 against 16.4 at 20,000. Below that, and for rows that are not aligned, one
// tile per block: 32 columns while all blocks are resident at once, else 64 by 8-byte loads (20,242 columns, both halves of a
// working set inside a solve: 27 us in one and a half rounds of blocks, 16.6 in one).
static tsvm_status launch_update_f(double *f, int n, const double *alpha_diff, int q, int first_half_phys, const float *rows,
                                   long long ld, int t0, int t_mid, int t1, const int *row_slot, cudaStream_t st,
                                   const StatusArgs &status = StatusArgs()) {
    const int wide_tiles = ceil_div(n, 128), sms = device_sm_count(), more = status.c != nullptr;
    if (((uintptr_t) rows & 15) == 0 && (ld & 3) == 0 && 2 * wide_tiles >= 3 * sms)
        TSVM_LAUNCH(update_f_kernel<4>, wide_tiles + more < UPD_WIDE_PER_SM * sms ? wide_tiles + more : UPD_WIDE_PER_SM * sms,
                    UPD_WARPS * 32, 0, st, f, n, alpha_diff, q, first_half_phys, rows, ld, t0, t_mid, t1, row_slot, status);
    else if (((uintptr_t) rows & 7) == 0 && (ld & 1) == 0 && ceil_div(n, 32) + more > UPD_NARROW_PER_SM * sms)
        TSVM_LAUNCH(update_f_kernel<2>, ceil_div(n, 64) + more, UPD_WARPS * 32, 0, st, f, n, alpha_diff, q, first_half_phys, rows,
                    ld, t0, t_mid, t1, row_slot, status);
    else
        TSVM_LAUNCH(update_f_kernel<1>, ceil_div(n, 32) + more, UPD_WARPS * 32, 0, st, f, n, alpha_diff, q, first_half_phys, rows,
                    ld, t0, t_mid, t1, row_slot, status);
    return TSVM_OK;
}

static tsvm_status launch_local_smo(int solver_kind, int ws, const float *kww, const float *diag_ws, const int *y_ws,
                                    const double *f_ws, double *alpha_ws, double *alpha_diff, double Cp, double Cn,
                                    double eps, int max_iter, double *diff, const int *ids, double *alpha_global,
                                    cudaStream_t st, const int *stop = nullptr, PhaseTimes *times = nullptr) {
    const bool nu = solver_kind != TSVM_SOLVER_C;
    // four warps at every size, one to eight slots per thread: with eight warps every one repeats the reductions and the
    // step next to another on its scheduler (1,024 slots, rows in L1: 0.74 against 0.93 us per iteration, 1.65 with sixteen).
    // Blocks below 256 slots are small enough for L1 to hold what is used again.
    constexpr int T = 128;
    const int ahead = ws >= 256;
#define SMO_LAUNCH(NU, S)                                                                                          \
    do {                                                                                                           \
        TSVM_ONCE_PER_DEVICE(TSVM_CUDA(cudaFuncSetAttribute(local_smo_kernel<NU, S, T>,                            \
                                                            cudaFuncAttributePreferredSharedMemoryCarveout,        \
                                                            cudaSharedmemCarveoutMaxL1)));                         \
        TSVM_LAUNCH((local_smo_kernel<NU, S, T>), 1, T + (NU ? 0 : 64), 0, st, ws, kww, diag_ws, y_ws, f_ws,        \
                    alpha_ws, alpha_diff, Cp, Cn, eps, max_iter, diff, ids, alpha_global, stop, ahead, times);     \
    } while (0)
#define SMO_CASE(S) do { if (nu) SMO_LAUNCH(true, S); else SMO_LAUNCH(false, S); } while (0)
    if (ws <= T) SMO_CASE(1); else if (ws <= 2 * T) SMO_CASE(2); else if (ws <= 4 * T) SMO_CASE(4); else SMO_CASE(8);
#undef SMO_CASE
#undef SMO_LAUNCH
    return TSVM_OK;
}

}  // namespace tsvm

using namespace tsvm;

// Bytes a solver may use for its row buffer / kernel-row cache: what tsvm_set_row_cache_bytes or the environment
// variable TSVM_ROW_CACHE_MB asked for, else 45 % of the device's memory (a fixed fraction of the total, not of
// what happens to be free, so that consecutive solvers of the same problem ask for the same block and get it
// back from the library's pool).
static long long g_row_cache_bytes = -1;
static size_t row_cache_budget() {
    if (g_row_cache_bytes >= 0) return (size_t) g_row_cache_bytes;
    if (const char *e = getenv("TSVM_ROW_CACHE_MB")) return (size_t) strtoull(e, nullptr, 10) << 20;
    return (size_t) ((double) device_memory_bytes() * 0.45);
}

struct tsvm_ws {
    int n_max = 0, ws_max = 0;
    SelectState *state = nullptr;   // zero between calls, like ticket
    int *hist = nullptr, *ticket = nullptr, *count = nullptr;
    unsigned long long *cand_h = nullptr;       // [4][SELECT_CAP]
    unsigned int *cand_l = nullptr;
    double *sorted_f = nullptr;                 // [4][ws_max]
    int *sorted_id = nullptr;
};

extern "C" {

void tsvm_set_row_cache_bytes(long long bytes) { g_row_cache_bytes = bytes; }

// (the state still has to be cleared, see clear_select_state)
static tsvm_status ws_alloc(int n_max, int ws_max, tsvm_ws **out) {
    tsvm_ws *w = new tsvm_ws;
    w->n_max = n_max; w->ws_max = ws_max;
    tsvm_status s = dev_alloc(&w->state, MAX_LISTS + 1);         // the ticket lies behind the lists
    if (s == TSVM_OK) s = dev_alloc(&w->hist, MAX_LISTS * RADIX_BINS);
    if (s == TSVM_OK) s = dev_alloc(&w->count, 1);
    if (s == TSVM_OK) s = dev_alloc(&w->cand_h, (size_t) MAX_LISTS * SELECT_CAP);
    if (s == TSVM_OK) s = dev_alloc(&w->cand_l, (size_t) MAX_LISTS * SELECT_CAP);
    if (s == TSVM_OK) s = dev_alloc(&w->sorted_f, (size_t) MAX_LISTS * ws_max);
    if (s == TSVM_OK) s = dev_alloc(&w->sorted_id, (size_t) MAX_LISTS * ws_max);
    if (s != TSVM_OK) { tsvm_ws_destroy(w); return s; }
    w->ticket = reinterpret_cast<int *>(w->state + MAX_LISTS);
    *out = w;
    return TSVM_OK;
}
static tsvm_status clear_select_state(tsvm_ws *w, cudaStream_t st) {
    TSVM_CUDA(cudaMemsetAsync(w->state, 0, (MAX_LISTS + 1) * sizeof(SelectState), st));
    return TSVM_OK;
}

tsvm_status tsvm_ws_create(int n_max, int ws_max, tsvm_ws **out) {
    TSVM_REQUIRE(out && n_max > 0 && ws_max > 0 && ws_max <= MERGE_MAX_WANT, "ws_create: bad arguments");
    *out = nullptr;
    tsvm_ws *w = nullptr;
    TSVM_TRY(ws_alloc(n_max, ws_max, &w));
    tsvm_status s = clear_select_state(w, nullptr);
    if (s == TSVM_OK && cudaStreamSynchronize(nullptr) != cudaSuccess) {     // the first call may be on any stream
        set_error("ws_create: clearing the selection state failed");
        s = TSVM_ERR_CUDA;
    }
    if (s != TSVM_OK) { tsvm_ws_destroy(w); return s; }
    *out = w;
    return TSVM_OK;
}

static void ws_destroy(tsvm_ws *w, bool idle) {
    if (!w) return;
    pool_free_many({w->state, w->hist, w->count, w->cand_h, w->cand_l, w->sorted_f, w->sorted_id}, idle);
    delete w;
}
void tsvm_ws_destroy(tsvm_ws *w) { ws_destroy(w, false); }

// The selection in one cooperative launch (select_kernel). out_ids: the merged selection; else the sorted lists
// ([lists][want], padding id -1) in sorted_f / sorted_id are the result.
static tsvm_status launch_select(tsvm_ws *w, int solver_kind, int n, const double *f_dev, const double *alpha_dev,
                                 const int *y_dev, const unsigned char *in_ws_dev, double Cp, double Cn, int want,
                                 int id_offset, double *sorted_f, int *sorted_id, int *out_ids, const int *stop,
                                 cudaStream_t st, PhaseTimes *times = nullptr) {
    const int lists = solver_kind == TSVM_SOLVER_C ? 2 : 4;
    static int resident_blocks[MAX_DEVICES] = {0};
    int dev = 0;
    TSVM_CUDA(cudaGetDevice(&dev));
    int &max_blocks = resident_blocks[dev & (MAX_DEVICES - 1)];
    if (!max_blocks) {
        TSVM_CUDA(cudaFuncSetAttribute(select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int) select_smem_bytes(MAX_LISTS, SAMPLE_MAX)));
        int sms = 0, coop = 0;
        TSVM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        TSVM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        TSVM_REQUIRE(coop, "working-set selection needs a device that supports cooperative launches");
        max_blocks = sms;                         // one 1024-thread block per SM: always resident together
    }
    SelectArgs a;
    a.solver_kind = solver_kind; a.n = n; a.f = f_dev; a.alpha = alpha_dev; a.y = y_dev; a.in_ws = in_ws_dev;
    a.Cp = Cp; a.Cn = Cn; a.st = w->state; a.hist = w->hist; a.ticket = w->ticket; a.want = want;
    a.id_offset = id_offset; a.cand_h = w->cand_h; a.cand_l = w->cand_l; a.sorted_f = sorted_f; a.sorted_id = sorted_id;
    a.out_ids = out_ids; a.out_count = w->count; a.stop = stop; a.times = times;
    a.sample = select_sample(n);
    if (a.sample == n) { a.rank_low = want; a.rank_high = want + want / 2; }
    else {
        // `want` instances put want * sample / n of their own into the sample, give or take the square root of that;
        // 3.2 of these and two more are added so that the pivot hardly ever falls short
        const double mean = (double) want * a.sample / n;
        a.rank_low = (int) (mean + 3.2 * sqrt(mean) + 2.0);
        a.rank_high = a.rank_low + a.rank_low / 4 + 2;
    }
    int grid = select_grid(n);
    if (grid > max_blocks) grid = max_blocks;
    void *args[] = {&a};
    TSVM_CUDA(cudaLaunchCooperativeKernel((const void *) select_kernel, dim3(grid), dim3(SELECT_THREADS), args,
                                          select_smem_bytes(lists, a.sample), st));
    count_launch();
    return TSVM_OK;
}

tsvm_status tsvm_ws_candidates(tsvm_ws *w, int solver_kind, int n, const double *f_dev, const double *alpha_dev,
                               const int *y_dev, const unsigned char *in_ws_dev, double Cp, double Cn, int want,
                               int id_offset, double *cand_f_dev, int *cand_id_dev, void *stream) {
    TSVM_REQUIRE(w && f_dev && alpha_dev && y_dev && cand_f_dev && cand_id_dev && n > 0 && want > 0 &&
                 want <= w->ws_max && solver_kind >= 0 && solver_kind <= 2, "ws_candidates: bad arguments");
    return launch_select(w, solver_kind, n, f_dev, alpha_dev, y_dev, in_ws_dev, Cp, Cn, want, id_offset, cand_f_dev,
                         cand_id_dev, nullptr, nullptr, (cudaStream_t) stream);
}

static tsvm_status ws_merge_impl(tsvm_ws *w, int solver_kind, const double *cand_f_dev, const int *cand_id_dev, int len,
                                 int seg_len, int want, int *out_ids_dev, cudaStream_t st) {
    const size_t smem = merge_smem_bytes(len);
    TSVM_ONCE_PER_DEVICE(TSVM_CUDA(cudaFuncSetAttribute(select_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int) merge_smem_bytes(MERGE_MAX_LEN))));
    TSVM_LAUNCH(select_merge_kernel, 1, MERGE_THREADS, smem, st, solver_kind, cand_f_dev, cand_id_dev, len, want,
                out_ids_dev, w->count, seg_len);
    return TSVM_OK;
}

tsvm_status tsvm_ws_merge(tsvm_ws *w, int solver_kind, const double *cand_f_dev, const int *cand_id_dev, int len,
                          int want, int *out_ids_dev, void *stream) {
    TSVM_REQUIRE(w && cand_f_dev && cand_id_dev && out_ids_dev && len > 0 && len <= MERGE_MAX_LEN && want > 0 &&
                 want <= MERGE_MAX_WANT, "ws_merge: bad arguments (len=%d want=%d)", len, want);
    return ws_merge_impl(w, solver_kind, cand_f_dev, cand_id_dev, len, 0, want, out_ids_dev, (cudaStream_t) stream);
}

static tsvm_status ws_sort_impl(int solver_kind, const double *in_f, const int *in_id, int len, double *out_f, int *out_id,
                                int out_len, cudaStream_t st) {
    int P = 1;
    while (P < len) P <<= 1;
    const size_t smem = (size_t) P * 12 + 8 + (size_t) P * 8;
    TSVM_ONCE_PER_DEVICE(TSVM_CUDA(cudaFuncSetAttribute(select_sort_candidates_kernel,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int) ((size_t) MERGE_MAX_LEN * 20 + 8))));
    TSVM_LAUNCH(select_sort_candidates_kernel, solver_kind == TSVM_SOLVER_C ? 2 : 4, MERGE_THREADS, smem, st,
                solver_kind, in_f, in_id, len, out_f, out_id, out_len);
    return TSVM_OK;
}

tsvm_status tsvm_ws_sort_candidates(tsvm_ws *w, int solver_kind, double *cand_f_dev, int *cand_id_dev, int len,
                                    void *stream) {
    TSVM_REQUIRE(w && cand_f_dev && cand_id_dev && len > 0 && len <= MERGE_MAX_LEN && solver_kind >= 0 &&
                 solver_kind <= 2, "ws_sort_candidates: bad arguments (len=%d)", len);
    return ws_sort_impl(solver_kind, cand_f_dev, cand_id_dev, len, cand_f_dev, cand_id_dev, len, (cudaStream_t) stream);
}

tsvm_status tsvm_ws_merge_sorted(tsvm_ws *w, int solver_kind, const double *cand_f_dev, const int *cand_id_dev, int len,
                                 int seg_len, int want, int *out_ids_dev, void *stream) {
    TSVM_REQUIRE(w && cand_f_dev && cand_id_dev && out_ids_dev && len > 0 && len <= MERGE_MAX_LEN && want > 0 &&
                 want <= MERGE_MAX_WANT && seg_len > 0 && len % seg_len == 0 && len / seg_len <= MERGE_THREADS,
                 "ws_merge_sorted: bad arguments (len=%d seg_len=%d want=%d)", len, seg_len, want);
    return ws_merge_impl(w, solver_kind, cand_f_dev, cand_id_dev, len, seg_len, want, out_ids_dev, (cudaStream_t) stream);
}

tsvm_status tsvm_select_working_set(tsvm_ws *w, int solver_kind, int n, const double *f_dev, const double *alpha_dev,
                                    const int *y_dev, const unsigned char *in_ws_dev, double Cp, double Cn, int want,
                                    int *out_ids_dev, void *stream) {
    TSVM_REQUIRE(w && f_dev && alpha_dev && y_dev && out_ids_dev && n > 0 && want > 0 && want <= w->ws_max &&
                 solver_kind >= 0 && solver_kind <= 2, "select_working_set: bad arguments");
    return launch_select(w, solver_kind, n, f_dev, alpha_dev, y_dev, in_ws_dev, Cp, Cn, want, 0, w->sorted_f, w->sorted_id,
                         out_ids_dev, nullptr, (cudaStream_t) stream);
}

// ---- working-set selection without any allocation --------------------------------------------------
// Scratch of tsvm_select_working_set_static: the per-list selection state, the radix histograms, the
// ticket / count words and the candidate lists for up to TSVM_STATIC_WS_MAX wanted ids and four
// lists. It is a fixed part of the library image: every GPU that loads the library holds these
// bytes until the process exits.
constexpr int STATIC_WS_MAX = TSVM_STATIC_WS_MAX;
constexpr size_t STATIC_OFF_STATE = 0;                                                   // SelectState[4]
constexpr size_t STATIC_OFF_HIST = 256;                                                  // int[4 * 4096]
constexpr size_t STATIC_OFF_TICKET = STATIC_OFF_HIST + sizeof(int) * MAX_LISTS * RADIX_BINS;   // int
constexpr size_t STATIC_OFF_COUNT = STATIC_OFF_TICKET + 128;                             // int
constexpr size_t STATIC_OFF_CAND_H = STATIC_OFF_COUNT + 128;                             // uint64[4 * SELECT_CAP]
constexpr size_t STATIC_OFF_CAND_L = STATIC_OFF_CAND_H + 8 * MAX_LISTS * SELECT_CAP;     // uint32[4 * SELECT_CAP]
constexpr size_t STATIC_OFF_SORTED_F = STATIC_OFF_CAND_L + 4 * MAX_LISTS * SELECT_CAP;   // double[4 * 1024]
constexpr size_t STATIC_OFF_SORTED_ID = STATIC_OFF_SORTED_F + sizeof(double) * MAX_LISTS * STATIC_WS_MAX;
constexpr size_t STATIC_SCRATCH_BYTES = STATIC_OFF_SORTED_ID + sizeof(int) * MAX_LISTS * STATIC_WS_MAX;
static_assert(sizeof(SelectState) * MAX_LISTS <= STATIC_OFF_HIST, "selection state does not fit its slot");
static __device__ __align__(256) unsigned char g_static_select_scratch[STATIC_SCRATCH_BYTES];

// In host code the array's name is only a stand-in for the symbol, not a device address: the address
// is asked from the runtime once per device (with that device current) and remembered. The cache is
// written without a lock by whichever host thread calls first on a device; every writer stores the same
// value, so concurrent first calls are harmless.
constexpr int STATIC_MAX_DEVICES = MAX_DEVICES;
static unsigned char *g_static_scratch_addr[STATIC_MAX_DEVICES] = {nullptr};

tsvm_status tsvm_select_working_set_static(int solver_kind, int n, const double *f_dev, const double *alpha_dev,
                                           const int *y_dev, const unsigned char *in_ws_dev, double Cp, double Cn,
                                           int want, int *out_ids_dev, void *stream) {
    TSVM_REQUIRE(f_dev && alpha_dev && y_dev && out_ids_dev && n > 0 && want > 0 && solver_kind >= 0 &&
                 solver_kind <= 2, "select_working_set_static: bad arguments");
    TSVM_REQUIRE(want <= STATIC_WS_MAX,
                 "select_working_set_static: %d ids wanted, the built-in scratch holds at most %d "
                 "(use tsvm_select_working_set with a tsvm_ws for more)", want, STATIC_WS_MAX);
    int dev = 0;
    TSVM_CUDA(cudaGetDevice(&dev));
    TSVM_REQUIRE(dev >= 0 && dev < STATIC_MAX_DEVICES, "select_working_set_static: device ordinal %d not supported", dev);
    if (!g_static_scratch_addr[dev]) {
        void *p = nullptr;
        TSVM_CUDA(cudaGetSymbolAddress(&p, g_static_select_scratch));
        g_static_scratch_addr[dev] = static_cast<unsigned char *>(p);
    }
    unsigned char *base = g_static_scratch_addr[dev];
    tsvm_ws view;                      // a view over the static array; owns nothing, frees nothing
    view.n_max = n;
    view.ws_max = STATIC_WS_MAX;
    view.state = reinterpret_cast<SelectState *>(base + STATIC_OFF_STATE);
    view.hist = reinterpret_cast<int *>(base + STATIC_OFF_HIST);
    view.ticket = reinterpret_cast<int *>(base + STATIC_OFF_TICKET);
    view.count = reinterpret_cast<int *>(base + STATIC_OFF_COUNT);
    view.cand_h = reinterpret_cast<unsigned long long *>(base + STATIC_OFF_CAND_H);
    view.cand_l = reinterpret_cast<unsigned int *>(base + STATIC_OFF_CAND_L);
    view.sorted_f = reinterpret_cast<double *>(base + STATIC_OFF_SORTED_F);
    view.sorted_id = reinterpret_cast<int *>(base + STATIC_OFF_SORTED_ID);
    // the counters that have to be zero at the start of a call are zero in the image and are cleared again by the last
    // block of every call; nothing else of an earlier call's contents is read.
    return tsvm_select_working_set(&view, solver_kind, n, f_dev, alpha_dev, y_dev, in_ws_dev, Cp, Cn, want,
                                   out_ids_dev, stream);
}

tsvm_status tsvm_local_smo(int solver_kind, int ws_size, const float *kww_dev, const float *diag_ws_dev,
                           const int *y_ws_dev, const double *f_ws_dev, double *alpha_ws_dev, double *alpha_diff_dev,
                           double Cp, double Cn, double eps, int max_iter, double *diff_dev, void *stream) {
    TSVM_REQUIRE(ws_size > 0 && ws_size <= 1024 && kww_dev && diag_ws_dev && y_ws_dev && f_ws_dev && alpha_ws_dev &&
                 alpha_diff_dev && diff_dev, "local_smo: bad arguments (ws=%d)", ws_size);
    return launch_local_smo(solver_kind, ws_size, kww_dev, diag_ws_dev, y_ws_dev, f_ws_dev, alpha_ws_dev,
                            alpha_diff_dev, Cp, Cn, eps, max_iter, diff_dev, nullptr, nullptr, (cudaStream_t) stream);
}

tsvm_status tsvm_rho_partials(int n, const double *f_dev, const double *alpha_dev, const int *y_dev, double Cp,
                              double Cn, double *out13_dev, void *stream) {
    TSVM_REQUIRE(n > 0 && f_dev && alpha_dev && y_dev && out13_dev, "rho_partials: bad arguments");
    TSVM_LAUNCH(rho_obj_kernel, 1, 1024, 0, (cudaStream_t) stream, n, f_dev, alpha_dev, y_dev, Cp, Cn, out13_dev);
    return TSVM_OK;
}

tsvm_status tsvm_update_f(double *f_dev, int n, const double *alpha_diff_dev, int ws_size, const float *rows_dev,
                          long long ld, void *stream) {
    TSVM_REQUIRE(f_dev && alpha_diff_dev && rows_dev && n > 0 && ws_size > 0 && ws_size <= 1024 && ld >= n,
                 "update_f: bad arguments (at most 1024 rows per call)");
    TSVM_TRY(launch_update_f(f_dev, n, alpha_diff_dev, 0, 0, rows_dev, ld, 0, 0, ws_size, nullptr, (cudaStream_t) stream));
    return TSVM_OK;
}

int tsvm_working_set_size(int n_instances, int n_features, size_t max_mem_bytes, size_t used_bytes) {
    if (max_mem_bytes < used_bytes) return -1;
    // max2power(x) = 2^floor(log2f(x)) (include/thundersvm/util/common.h:20-23)
    auto max2power = [](double x) -> long long { return (long long) exp2(floor(log2f((float) x))); };
    const size_t free_mem = max_mem_bytes - used_bytes;
    long long a = max2power((double) n_instances);
    long long b = max2power((double) (free_mem / sizeof(float) / ((size_t) n_instances + n_features)));
    if (b > 1024) b = 1024;
    return (int) (a < b ? a : b);
}

}  // extern "C"

// Solver state that persists across outer iterations.
// How many iterations are queued before the device has finished the first of them: enough that the next one is there when
// one ends (the host needs 30 - 60 us to queue an iteration, more with several solvers at a time); every one queued past
// the end of a solve is a no-op of some 20 us.
enum { MAX_QUEUED = 32 };
static int queued_iterations(int otherwise) {
    static const int k = [] {
        const char *e = getenv("TSVM_SYNC_EVERY");
        const int v = e ? atoi(e) : 0;
        return !e ? 0 : (v < 1 ? 1 : (v > MAX_QUEUED ? (int) MAX_QUEUED : v));
    }();
    return k ? k : otherwise;
}
static int queue_depth() { return queued_iterations(3); }
static int sync_every() { return queued_iterations(8); }          // shard solver: iterations between two reads of the verdict

// The second stream of a solver and its events. Creating them costs more than the rest of a small solve's set-up (a stream
// 0.2 - 2 ms), so a finished solver leaves them to the next one of the same device: 16 sets at most are kept, and
// tsvm_release_cached_memory destroys them. A set belongs to one solver at a time and is idle when it comes back.
struct SolverStreams {
    int dev = 0;
    cudaStream_t st2 = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_fork2 = nullptr, ev_join = nullptr;

    ~SolverStreams() {
        for (auto e : {ev_fork, ev_fork2, ev_join}) if (e) cudaEventDestroy(e);
        if (st2) cudaStreamDestroy(st2);
    }
    tsvm_status create() {
        TSVM_CUDA(cudaGetDevice(&dev));
        TSVM_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
        TSVM_CUDA(cudaEventCreateWithFlags(&ev_fork2, cudaEventDisableTiming));
        TSVM_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
        int lo_prio = 0, hi_prio = 0;
        TSVM_CUDA(cudaDeviceGetStreamPriorityRange(&lo_prio, &hi_prio));
        TSVM_CUDA(cudaStreamCreateWithPriority(&st2, cudaStreamNonBlocking, hi_prio));
        return TSVM_OK;
    }
};
namespace {
constexpr size_t MAX_STREAM_SETS = 16;
std::mutex &g_streams_mu = *new std::mutex;
auto &g_streams_free = *new std::vector<SolverStreams *>;

tsvm_status take_streams(SolverStreams **out) {
    int dev = 0;
    TSVM_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(g_streams_mu);
        for (size_t k = g_streams_free.size(); k-- > 0;)
            if (g_streams_free[k]->dev == dev) {
                *out = g_streams_free[k];
                g_streams_free.erase(g_streams_free.begin() + k);
                return TSVM_OK;
            }
    }
    SolverStreams *s = new SolverStreams;
    const tsvm_status r = s->create();
    if (r != TSVM_OK) { delete s; return r; }
    *out = s;
    return TSVM_OK;
}
// idle: nothing is pending on the set's stream
void give_streams(SolverStreams *s, bool idle) {
    if (!s) return;
    if (idle) {
        std::lock_guard<std::mutex> lk(g_streams_mu);
        if (g_streams_free.size() < MAX_STREAM_SETS) { g_streams_free.push_back(s); return; }
    }
    delete s;
}
}  // namespace
namespace tsvm {
void release_solver_streams() {
    std::lock_guard<std::mutex> lk(g_streams_mu);
    int cur = 0;
    const bool have = cudaGetDevice(&cur) == cudaSuccess;
    for (auto *s : g_streams_free) {
        cudaSetDevice(s->dev);
        delete s;
    }
    g_streams_free.clear();
    if (have) cudaSetDevice(cur);
}
}  // namespace tsvm

static inline void cpu_pause() {
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#endif
}

struct tsvm_solver {
    tsvm_km *km = nullptr;
    std::shared_ptr<char> storage_user;
    int kind = 0, ws = 0, q = 0, n = 0;
    const int *y = nullptr;
    double *alpha = nullptr, *f = nullptr;
    double eps = 0, Cp = 0, Cn = 0;
    long long ld = 0;
    cudaStream_t st = nullptr;
    // device buffers
    int *ids = nullptr, *y_ws = nullptr;
    float *rows = nullptr, *kww = nullptr, *diag_ws = nullptr;
    double *f_ws = nullptr, *a_ws = nullptr, *alpha_diff = nullptr, *diff = nullptr, *red = nullptr;
    unsigned char *in_ws = nullptr;
    tsvm_ws *sel = nullptr;
    double *diff_host = nullptr;
    // end-of-iteration state on the device, its pinned copy, and the events of the queued iterations
    SolverCtl *ctl = nullptr, *ctl_host = nullptr;
    SolverStreams *streams = nullptr;
    bool idle = true;               // nothing of this solver is in flight (the last call ended with a wait)
    int max_iter = -1;              // iteration cap applied on the device; -1: none
    bool stopped = false;           // the device stopped the queue (done, capped or an error)
    bool uncollected = false;       // iterations have run since the control block was last copied back
    long long iter_collected = 0;   // iterations as of then
    // overlapped iteration: second stream, fork / join events, operand planes of the working set
    bool overlap = true;
    cudaStream_t st2 = nullptr;     // of `streams`, like the events
    cudaEvent_t ev_fork = nullptr, ev_fork2 = nullptr, ev_join = nullptr;
    float *ws_hi = nullptr, *ws_lo = nullptr, *ws_sd = nullptr, *ws_unscale = nullptr;
    // kernel-row cache (cache_assign_kernel): the row buffer holds cache_cap rows; directory and per-iteration lists
    long long cache_cap = 0;
    int *slot_of = nullptr, *inst_of = nullptr, *stamp = nullptr, *row_slots = nullptr, *miss_ids = nullptr,
        *miss_slot = nullptr, *victims = nullptr;
    long long *cache_ctr = nullptr;
    float *miss_hi = nullptr, *miss_lo = nullptr, *miss_sd = nullptr, *miss_unscale = nullptr;
    long long hits = 0, misses = 0, row_blocks = 0, row_blocks_saved = 0;
    // iteration state (csmosolver.cpp:51-57)
    long long iter = 0, local_iter = 0, rows_made = 0, launches0 = 0;
    int local_max_iter = 0;
    double diff0 = 0;
    double t_sel = 0, t_rows = 0, t_loc = 0, t_upd = 0;
    bool done = false;
    std::chrono::steady_clock::time_point t_begin;

    ~tsvm_solver() {
        pool_free_many({ids, y_ws, rows, kww, diag_ws, f_ws, a_ws, alpha_diff, diff, red, in_ws, ws_hi, ws_lo, ws_sd,
                        ws_unscale, slot_of, inst_of, stamp, row_slots, miss_ids, miss_slot, victims, cache_ctr, miss_hi,
                        miss_lo, miss_sd, miss_unscale, ctl}, idle);
        ws_destroy(sel, idle);
        if (diff_host) pinned_free(diff_host);
        if (ctl_host) pinned_free(ctl_host);
        give_streams(streams, idle);
    }

    tsvm_status ensure_ws_planes() {
        if (ws_hi) return TSVM_OK;
        const size_t words = (km_plane_row_bytes(km) * (size_t) ws + 3) / 4;
        TSVM_TRY(dev_alloc(&ws_hi, words));
        TSVM_TRY(dev_alloc(&ws_lo, words));
        TSVM_TRY(dev_alloc(&ws_sd, (size_t) ws));
        TSVM_TRY(dev_alloc(&ws_unscale, (size_t) ws));
        return TSVM_OK;
    }

    tsvm_status ensure_miss_planes() {
        if (miss_hi) return TSVM_OK;
        const size_t words = (km_plane_row_bytes(km) * (size_t) ws + 3) / 4;
        TSVM_TRY(dev_alloc(&miss_hi, words));
        TSVM_TRY(dev_alloc(&miss_lo, words));
        TSVM_TRY(dev_alloc(&miss_sd, (size_t) ws));
        TSVM_TRY(dev_alloc(&miss_unscale, (size_t) ws));
        return TSVM_OK;
    }

    // Row buffer = kernel-row cache: as many rows as the budget allows (tsvm_set_row_cache_bytes), at least the
    // working set plus one batch of new rows, at most one row per instance. A failed allocation halves the request, and so
    // does one that leaves no room for the solve's other buffers (looked at only after a failure: the device is nearly full).
    bool room_for_the_rest() const {
        const size_t staged = km->dense ? (size_t) 8 * km->d_pad : (size_t) km->d;        // floats per working-set member
        void *probe = nullptr;
        if (pool_alloc(&probe, ((size_t) 16 << 20) + sizeof(float) * ((size_t) (ws > 128 ? ws : 128) * (staged + ws) + (size_t) 8 * n)) != TSVM_OK)
            return false;
        pool_free_many({probe}, true);
        return true;
    }
    tsvm_status alloc_rows() {
        const long long floor_rows = (long long) ws + q;
        long long want = (long long) (row_cache_budget() / (sizeof(float) * (size_t) ld));
        if (want > n) want = n;
        if (want < floor_rows) want = floor_rows;
        km_pair_engine(km, st);                  // (operand planes that found no room before are built first)
        for (const long long first = want;;) {
            tsvm_status s = dev_alloc(&rows, (size_t) want * ld);
            if (s == TSVM_OK && want < first && want > floor_rows && !room_for_the_rest()) {
                pool_free_many({rows}, true);
                rows = nullptr;
                s = TSVM_ERR_OOM;
            }
            if (s == TSVM_OK) break;
            if (s != TSVM_ERR_OOM || want == floor_rows) return s;
            want = want / 2 > floor_rows ? want / 2 : floor_rows;
        }
        cache_cap = want;
        TSVM_TRY(dev_alloc(&slot_of, (size_t) n));
        TSVM_TRY(dev_alloc(&inst_of, (size_t) cache_cap));
        TSVM_TRY(dev_alloc(&stamp, (size_t) cache_cap));
        TSVM_TRY(dev_alloc(&row_slots, (size_t) 2 * ws));      // this iteration's and the previous one's
        TSVM_TRY(dev_alloc(&miss_ids, (size_t) ws));
        TSVM_TRY(dev_alloc(&miss_slot, (size_t) ws));
        TSVM_TRY(dev_alloc(&victims, (size_t) ws));
        TSVM_TRY(dev_alloc(&cache_ctr, (size_t) CACHE_CTRS));
        const int blocks = 2 * device_sm_count();
        TSVM_LAUNCH(fill_int_kernel, blocks, 256, 0, st, slot_of, (long long) n, -1);
        TSVM_LAUNCH(fill_int_kernel, blocks, 256, 0, st, inst_of, cache_cap, -1);
        TSVM_CUDA(cudaMemsetAsync(stamp, 0, sizeof(int) * (size_t) cache_cap, st));
        TSVM_CUDA(cudaMemsetAsync(row_slots, 0, sizeof(int) * (size_t) 2 * ws, st));
        TSVM_CUDA(cudaMemsetAsync(cache_ctr, 0, sizeof(long long) * CACHE_CTRS, st));
        return TSVM_OK;
    }

    tsvm_status allocate() {
        idle = false;
        TSVM_TRY(dev_alloc(&ids, (size_t) ws));
        TSVM_TRY(dev_alloc(&y_ws, (size_t) ws));
        TSVM_TRY(alloc_rows());
        TSVM_TRY(dev_alloc(&kww, (size_t) ws * ws));
        TSVM_TRY(dev_alloc(&diag_ws, (size_t) ws));
        TSVM_TRY(dev_alloc(&f_ws, (size_t) ws));
        TSVM_TRY(dev_alloc(&a_ws, (size_t) ws));
        TSVM_TRY(dev_alloc(&alpha_diff, (size_t) ws));
        TSVM_TRY(dev_alloc(&diff, 4));
        TSVM_TRY(dev_alloc(&red, 16));   // >= RHO_VALS
        TSVM_TRY(dev_alloc(&in_ws, (size_t) n));
        TSVM_CUDA(cudaMemsetAsync(in_ws, 0, (size_t) n, st));
        TSVM_TRY(ws_alloc(n, ws, &sel));
        TSVM_TRY(clear_select_state(sel, st));
        TSVM_TRY(pinned_alloc((void **) &diff_host, 16 * sizeof(double)));
        TSVM_TRY(dev_alloc(&ctl, 1));
        TSVM_TRY(pinned_alloc((void **) &ctl_host, sizeof(SolverCtl)));
        memset(ctl_host, 0, sizeof(SolverCtl));
        *progress() = 0;
        ctl_host->prev = ctl_host->last = ctl_host->second_last = INFINITY;     // csmosolver.cpp:51-57
        TSVM_CUDA(cudaMemcpyAsync(ctl, ctl_host, sizeof(SolverCtl), cudaMemcpyHostToDevice, st));
        TSVM_TRY(take_streams(&streams));
        st2 = streams->st2; ev_fork = streams->ev_fork; ev_fork2 = streams->ev_fork2; ev_join = streams->ev_join;
        // local iteration cap: max(100000, 100 * ws) (csmosolver.cpp:49)
        local_max_iter = ws > INT_MAX / 100 ? INT_MAX : (100 * ws > 100000 ? 100 * ws : 100000);
        return TSVM_OK;
    }

    // init_f (csmosolver.cpp:189-214): f -= sum over the initially non-zero alphas
    tsvm_status init_f() {
        // all zero, as C-SVC starts: nothing to add, and no need for the alphas on the host
        int *nonzero = reinterpret_cast<int *>(red);
        TSVM_CUDA(cudaMemsetAsync(nonzero, 0, sizeof(int), st));
        const int blocks = 2 * device_sm_count();
        TSVM_LAUNCH(any_nonzero_kernel, ceil_div(n, 4096) < blocks ? ceil_div(n, 4096) : blocks, 256, 0, st, alpha, n, nonzero);
        TSVM_CUDA(cudaMemcpyAsync(diff_host, nonzero, sizeof(int), cudaMemcpyDeviceToHost, st));
        TSVM_CUDA(cudaStreamSynchronize(st));
        if (*reinterpret_cast<const int *>(diff_host) == 0) { idle = true; return TSVM_OK; }
        std::vector<double> a_h(n);
        std::vector<int> y_h(n);
        TSVM_CUDA(cudaMemcpyAsync(a_h.data(), alpha, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
        TSVM_CUDA(cudaMemcpyAsync(y_h.data(), y, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
        TSVM_CUDA(cudaStreamSynchronize(st));
        std::vector<int> bi;
        std::vector<double> bd;
        auto flush = [&]() -> tsvm_status {
            if (bi.empty()) return TSVM_OK;
            const int m = (int) bi.size();
            TSVM_CUDA(cudaMemcpyAsync(ids, bi.data(), sizeof(int) * m, cudaMemcpyHostToDevice, st));
            TSVM_CUDA(cudaMemcpyAsync(alpha_diff, bd.data(), sizeof(double) * m, cudaMemcpyHostToDevice, st));
            TSVM_TRY(tsvm_km_rows_by_index(km, ids, m, rows, ld, st));
            TSVM_TRY(launch_update_f(f, n, alpha_diff, 0, 0, rows, ld, 0, 0, m, nullptr, st));
            TSVM_CUDA(cudaStreamSynchronize(st));
            rows_made += m;
            bi.clear(); bd.clear();
            return TSVM_OK;
        };
        for (int i = 0; i < n; ++i) {
            if (a_h[i] != 0) { bi.push_back(i); bd.push_back(-a_h[i] * y_h[i]); }
            if ((int) bi.size() == ws) TSVM_TRY(flush());
        }
        TSVM_TRY(flush());
        idle = true;
        return TSVM_OK;
    }

    // Queues one outer iteration of csmosolver.cpp:59-120, number `it`, without waiting for it. Its last launch
    // applies the reference's termination rules (csmosolver.cpp:86-111) on the device; every launch of an
    // iteration queued after the one that ended the solve is a no-op.
    //
    // Overlapped form (dense data on the CTA-pair tensor engine, every iteration but the first): the local
    // solver only needs the ws x ws block of kernel values, not the q full rows. The block's q new rows are
    // computed first by a small launch of the same engine against the working set's own operand planes
    // (bit-identical to the values the full rows will hold: same planes, same slab order), its old rows are
    // gathered from the rows already in the buffer, and the one-CTA local solver then runs on a second stream
    // while the q x n launch - which leaves one SM pair free for it - fills the row buffer. Both meet before
    // the f update.
    tsvm_status enqueue_iteration(long long it) {
        const int t0 = it == 0 ? 0 : q, n_new = it == 0 ? ws : q;          // iteration 0 fills the whole working set
        const bool overlapped = overlap && it > 0 && st2 && km_pair_engine(km, st);
        const int row_block = km_pair_engine(km, st) ? 256 : 64;           // requested rows per tile of the engine
        const int *n_miss_dev = reinterpret_cast<const int *>(cache_ctr);
        const int *stop = &ctl->stop;
        PhaseTimes *times = &ctl->times;
        int *row_slot = row_slots + (it & 1) * ws;                         // row of every working-set slot
        const int *row_slot_before = row_slots + ((it + 1) & 1) * ws;
        // (the status kernel of the previous iteration has rotated the working set)
        TSVM_TRY(launch_select(sel, kind, n, f, alpha, y, it == 0 ? nullptr : in_ws, Cp, Cn, n_new, 0, sel->sorted_f,
                               sel->sorted_id, ids + t0, it == 0 ? nullptr : stop, st, times));
        if (overlapped) {
            // The block needs the members' planes and the old members' rows, both known now: the second stream starts on
            // it while the first one still runs the cache directory, i.e. before the big launch takes all SM pairs
            // but one (started after it, the gather alone took 240 us at 200,000 instances; now 20). Rows 0..q-1 come
            // from the row buffer (where the previous iteration left them), rows q..ws-1 are computed from the members' own
            // operand planes.
            TSVM_TRY(ensure_ws_planes());
            TSVM_TRY(ensure_miss_planes());
            TSVM_TRY(km_gather_planes(km, ids, ws, nullptr, ws_hi, ws_lo, ws_sd, ws_unscale, st));
            TSVM_CUDA(cudaEventRecord(ev_fork, st));
            TSVM_CUDA(cudaStreamWaitEvent(st2, ev_fork, 0));
            TSVM_LAUNCH(gather_ws_kernel, ws, 256, 0, st2, ws, q, 0, ids, rows, ld, km->diag, y, f, alpha, kww, diag_ws,
                        y_ws, f_ws, a_ws, q, row_slot_before + q, (PhaseTimes *) nullptr);
            const size_t rb = km_plane_row_bytes(km);
            const InstancePlanes members{ws_hi, ws_lo, ws_sd, ws_unscale, ws};
            const RowPlanes new_members{reinterpret_cast<const float *>(reinterpret_cast<const char *>(ws_hi) + (size_t) q * rb),
                                        reinterpret_cast<const float *>(reinterpret_cast<const char *>(ws_lo) + (size_t) q * rb),
                                        ws_sd + q, ws_unscale + q};
            // (spread over all SM pairs it is done sooner, but the big launch waits for them: with more than four rounds of
            // tiles that one is the longer path, 200,000 x 2,000 457 ms per solve against 460)
            km->whole_blocks = (long long) ceil_div(n, 256) * ceil_div(q, 256) > 4 * (device_sm_count() / 2);
            const tsvm_status bs = km_rows_planes_on(km, members, new_members, q, kww + (size_t) q * ws, ws, st2);
            km->whole_blocks = false;
            TSVM_TRY(bs);
            TSVM_TRY(launch_local_smo(kind, ws, kww, diag_ws, y_ws, f_ws, a_ws, alpha_diff, Cp, Cn, eps, local_max_iter,
                                      diff, ids, alpha, st2, stop, times));
        }
        // cache directory: hits point at their rows, misses get the least recently used rows
        TSVM_LAUNCH(cache_assign_kernel, 1, CACHE_THREADS, 0, st, ids, t0, n_new, (int) (it + 1), slot_of, inst_of, stamp,
                    (int) cache_cap, row_slot_before, row_slot, miss_ids, miss_slot, victims, cache_ctr, row_block, stop, times);
        if (!overlapped) {
            // the engine computes the missing rows only (their number is read on the device) into their cache rows
            km->rows_m_dev = n_miss_dev; km->rows_slot_dev = miss_slot;
            const tsvm_status rs = tsvm_km_rows_by_index(km, miss_ids, n_new, rows, ld, st);
            km->rows_m_dev = nullptr; km->rows_slot_dev = nullptr;
            TSVM_TRY(rs);
        } else {
            TSVM_TRY(km_gather_planes(km, miss_ids, q, n_miss_dev, miss_hi, miss_lo, miss_sd, miss_unscale, st));
            TSVM_CUDA(cudaEventRecord(ev_fork2, st));
            TSVM_CUDA(cudaStreamWaitEvent(st2, ev_fork2, 0));
            // the rows that were in the buffer already can be applied to f at once (HBM-bound, next to the
            // tensor-bound launch); the new rows follow on the first stream
            TSVM_TRY(launch_update_f(f, n, alpha_diff, q, 0, rows, ld, 0, 0, q, row_slot, st2));
            TSVM_CUDA(cudaEventRecord(ev_join, st2));
            // first stream: the missing rows against all instances, on all SM pairs but one
            const InstancePlanes all{km->Xhi, km->Xlo, km->self_dot, km->x_unscale, km->n};
            const RowPlanes miss_rows{miss_hi, miss_lo, miss_sd, miss_unscale};
            km->reserve_clusters = 1;
            km->rows_m_dev = n_miss_dev; km->rows_slot_dev = miss_slot; km->rows_end_dev = &times->rows_end;
            const tsvm_status rs = km_rows_planes_on(km, all, miss_rows, q, rows, ld, st);
            km->reserve_clusters = 0;
            km->rows_m_dev = nullptr; km->rows_slot_dev = nullptr; km->rows_end_dev = nullptr;
            TSVM_TRY(rs);
        }
        if (!overlapped) {
            TSVM_LAUNCH(gather_ws_kernel, ws, 256, 0, st, ws, q, 0, ids, rows, ld, km->diag, y, f, alpha, kww, diag_ws,
                        y_ws, f_ws, a_ws, ws, row_slot, times);
            TSVM_TRY(launch_local_smo(kind, ws, kww, diag_ws, y_ws, f_ws, a_ws, alpha_diff, Cp, Cn, eps, local_max_iter,
                                      diff, ids, alpha, st, stop, times));
        } else {
            TSVM_CUDA(cudaStreamWaitEvent(st, ev_join, 0));
        }
        // f -= sum over the old half's rows, then f -= sum over the new half's rows: two sums in every form of the iteration,
        // so that all of them round alike (the first iteration has new rows only; overlapped, the old half is done)
        StatusArgs status;
        status.c = ctl; status.diff = diff; status.got = sel->count; status.wanted = n_new; status.eps = eps; status.max_iter = max_iter;
        status.cache_ctr = cache_ctr; status.engine_status = km->status_dev; status.ids = ids; status.q = q; status.in_ws = in_ws;
        status.progress = progress(); status.parity = (int) (it & 1);
        TSVM_TRY(launch_update_f(f, n, alpha_diff, q, 0, rows, ld, overlapped ? q : 0, it == 0 ? 0 : q, ws, row_slot, st, status));
        return TSVM_OK;
    }


    // Up to `count` outer iterations; fewer if the termination rules, the iteration cap or an error stop the queue on the
    // device. The device tells after every iteration how far it is, and the host keeps `queue_depth()` iterations queued:
    // there is always one ready when another ends, and few no-op ones follow the last. collect() has to come next.
    tsvm_status run_iterations(int count) {
        const long long end = iter + count;
        long long queued = iter;
        idle = false;
        uncollected = true;
        km->launched(st);                // (the overlapped iteration reads the handle's planes by itself); collect() ends it
        while (!stopped && iter < end) {
            const int ahead = iter == 0 ? 1 : queue_depth();      // (many small solves end with their first iteration)
            while (queued < end && queued < iter + ahead) TSVM_TRY(enqueue_iteration(queued++));
            TSVM_TRY(await_progress());
        }
        return TSVM_OK;
    }

    volatile unsigned long long *progress() const { return reinterpret_cast<volatile unsigned long long *>(diff_host + 15); }

    // Waits until the device has finished more iterations than `iter`, or has stopped.
    tsvm_status await_progress() {
        for (unsigned k = 1;; ++k) {
            const unsigned long long p = *progress();
            if ((long long) (p >> 1) > iter || (p & 1)) {
                iter = (long long) (p >> 1);
                stopped = (p & 1) != 0;
                return TSVM_OK;
            }
            if (k & 255) { cpu_pause(); continue; }
            const cudaError_t e = cudaStreamQuery(st);            // a failed launch or kernel makes no progress
            if (e == cudaErrorNotReady) { cudaGetLastError(); sched_yield(); continue; }
            TSVM_CUDA(e);
            const unsigned long long last = *progress();
            TSVM_REQUIRE((long long) (last >> 1) > iter || (last & 1), "solver: the queue ended without progress");
        }
    }

    // Waits for the queue and takes over what the device decided. `more`: enqueues further copies to wait for as well.
    template <typename More> tsvm_status collect(More more) {
        if (uncollected) TSVM_CUDA(cudaMemcpyAsync(ctl_host, ctl, sizeof(SolverCtl), cudaMemcpyDeviceToHost, st));
        TSVM_TRY(more());
        TSVM_CUDA(cudaStreamSynchronize(st));            // (the second stream has joined the first)
        idle = true;
        km->waited(st);
        if (!uncollected) return TSVM_OK;
        uncollected = false;
        const SolverCtl &c = *ctl_host;
        if (c.engine_status != 0) {
            set_error("dense kernel-row engine reported status %d (a bounded wait ran out)", c.engine_status);
            return TSVM_ERR_DEVICE;
        }
        t_sel = c.ns_select * 1e-9; t_rows = c.ns_rows * 1e-9; t_loc = c.ns_local * 1e-9; t_upd = c.ns_update * 1e-9;
        const long long last_end = c.update_end[0] > c.update_end[1] ? c.update_end[0] : c.update_end[1];
        if (c.update_begin && last_end > c.update_begin) t_upd += (last_end - c.update_begin) * 1e-9;       // (of the last iteration)
        hits = c.ctr[CACHE_HITS]; misses = c.ctr[CACHE_MISSES];
        row_blocks = c.ctr[CACHE_BLOCKS]; row_blocks_saved = c.ctr[CACHE_BLOCKS_SAVED];
        rows_made += (c.iter - iter_collected) * q + (iter_collected == 0 && c.iter > 0 ? ws - q : 0);
        iter = iter_collected = c.iter;
        local_iter = c.local_iter;
        diff0 = c.diff0;
        done = c.done != 0;
        stopped = c.stop != 0;
        if (c.short_wanted > 0) {
            // the reference's selection loop never ends here (csmosolver.cpp:131-164); the empty slots were inert
            set_error("working-set selection found %d eligible instances for %d slots (is a class weight or C zero?)",
                      c.short_got, c.short_wanted);
            return TSVM_ERR_INVALID;
        }
        return TSVM_OK;
    }
    tsvm_status collect() { return collect([] { return TSVM_OK; }); }

    void fill_stats(tsvm_solve_stats *out, double obj) const {
        out->outer_iters = iter;
        out->local_iters = local_iter;
        out->final_diff = diff0;
        out->objective = obj;
        out->seconds_select = t_sel;
        out->seconds_rows = t_rows;
        out->seconds_local = t_loc;
        out->seconds_update = t_upd;
        out->seconds_total = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_begin).count();
        out->kernel_rows = rows_made;
        out->gpu_launches = launch_count() - launches0;
        out->cache_hits = hits;
        out->cache_misses = misses;
        out->cache_rows = cache_cap;
        out->row_blocks = row_blocks;
        out->row_blocks_saved = row_blocks_saved;
    }

    // rho and objective (csmosolver.cpp:167-187,227-239; nusmosolver.cpp:9-46,120-126)
    tsvm_status finish(double *rho_host, tsvm_solve_stats *stats_host) {
        idle = false;
        TSVM_LAUNCH(rho_obj_kernel, 1, 1024, 0, st, n, f, alpha, y, Cp, Cn, red);
        TSVM_TRY(collect([&]() -> tsvm_status {
            TSVM_CUDA(cudaMemcpyAsync(diff_host, red, RHO_VALS * sizeof(double), cudaMemcpyDeviceToHost, st));
            return TSVM_OK;
        }));
        const double *R = diff_host;
        const double obj = -R[4];
        double rho;
        if (kind == TSVM_SOLVER_C) {
            const double nfree = R[0] + R[2];
            rho = nfree != 0 ? (R[1] + R[3]) / nfree : -(fmin(R[5], R[7]) + fmax(R[6], R[8])) / 2;
        } else {
            // nusmosolver.cpp:9-46 works with -f: r = -(min_{I_up}(-f) + max_{I_low}(-f)) / 2
            //                                       =  (max_{I_up} f + min_{I_low} f) / 2
            const double r1 = R[0] != 0 ? R[1] / R[0] : (R[9] + R[10]) / 2;
            const double r2 = R[2] != 0 ? -R[3] / R[2] : (R[11] + R[12]) / 2;
            rho = (r1 - r2) / 2;
            if (kind == TSVM_SOLVER_NU_SVC) {
                const double r = (r1 + r2) / 2;
                TSVM_LAUNCH(scale_kernel, ceil_div(n, 256), 256, 0, st, alpha, n, r);
                idle = false;
                TSVM_CUDA(cudaStreamSynchronize(st));
                rho /= r;
            }
        }
        idle = true;
        *rho_host = rho;
        if (stats_host) fill_stats(stats_host, obj);
        return TSVM_OK;
    }
};

extern "C" {

// ---- the solver as an object: create / iterate / finish -------------------------------------------
tsvm_status tsvm_solver_create(tsvm_km *km, int solver_kind, const int *y_dev, double *alpha_dev, double *f_dev,
                               double eps, double Cp, double Cn, int ws_size, void *stream, tsvm_solver **out) {
    TSVM_REQUIRE(out && km && y_dev && alpha_dev && f_dev, "solver_create: null argument");
    TSVM_REQUIRE(solver_kind >= 0 && solver_kind <= 2, "solver_create: unknown solver %d", solver_kind);
    const int n = km->n;
    TSVM_REQUIRE(ws_size >= 2 && ws_size <= 1024 && ws_size <= n && (ws_size & (ws_size - 1)) == 0,
                 "solver_create: working-set size %d must be a power of two in [2, min(n, 1024)]", ws_size);
    *out = nullptr;
    for (;;) {
        tsvm_solver *S = new tsvm_solver;
        S->km = km; S->storage_user = km->storage_users;
        S->kind = solver_kind; S->y = y_dev; S->alpha = alpha_dev; S->f = f_dev;
        S->eps = eps; S->Cp = Cp; S->Cn = Cn; S->ws = ws_size; S->q = ws_size / 2; S->n = n;
        S->ld = ((long long) n + 3) & ~3ll;
        S->st = (cudaStream_t) stream;
        S->launches0 = launch_count();
        S->t_begin = std::chrono::steady_clock::now();
        const tsvm_status s = S->allocate();
        const tsvm_status r = s == TSVM_OK ? S->init_f() : s;
        if (r == TSVM_OK) { *out = S; return TSVM_OK; }
        delete S;
        // a dense copy of CSR data makes the solve faster, but a solve without it is better than none
        if (s != TSVM_ERR_OOM || !km->from_csr || km->storage_users.use_count() > 1) return r;
        km_drop_dense_copy(km);
    }
}

tsvm_status tsvm_solver_iterate(tsvm_solver *S, int n_iters, int *done_host) {
    TSVM_REQUIRE(S && n_iters > 0, "solver_iterate: bad arguments");
    if (!S->done) {
        S->stopped = false;              // (an error may have ended the last call; the device says so again)
        TSVM_TRY(S->run_iterations(n_iters));
        TSVM_TRY(S->collect());
    }
    if (done_host) *done_host = S->done ? 1 : 0;
    return TSVM_OK;
}

tsvm_status tsvm_solver_finish(tsvm_solver *S, double *rho_host, tsvm_solve_stats *stats_host) {
    TSVM_REQUIRE(S && rho_host, "solver_finish: null argument");
    return S->finish(rho_host, stats_host);
}

tsvm_status tsvm_solver_get_stats(const tsvm_solver *S, tsvm_solve_stats *stats_host) {
    TSVM_REQUIRE(S && stats_host, "solver_get_stats: null argument");
    S->fill_stats(stats_host, NAN);
    return TSVM_OK;
}

tsvm_status tsvm_solver_set_overlap(tsvm_solver *S, int enable) {
    TSVM_REQUIRE(S, "solver_set_overlap: null argument");
    S->overlap = enable != 0;
    return TSVM_OK;
}

void tsvm_solver_destroy(tsvm_solver *S) { delete S; }

tsvm_status tsvm_smo_solve(tsvm_km *km, int solver_kind, const int *y_dev, double *alpha_dev, double *f_dev,
                           double eps, double Cp, double Cn, int ws_size, int max_iter, double *rho_host,
                           tsvm_solve_stats *stats_host, void *stream) {
    TSVM_REQUIRE(rho_host, "smo_solve: null argument");
    tsvm_solver *S = nullptr;
    TSVM_TRY(tsvm_solver_create(km, solver_kind, y_dev, alpha_dev, f_dev, eps, Cp, Cn, ws_size, stream, &S));
    tsvm_status s = TSVM_OK;
    // max_iter = k stops after outer iteration k, i.e. k + 1 iterations (csmosolver.cpp:110); applied on the device
    S->max_iter = max_iter;
    while (s == TSVM_OK && !S->stopped) s = S->run_iterations(INT_MAX);
    if (s == TSVM_OK) s = S->finish(rho_host, stats_host);
    delete S;
    return s;
}

}  // extern "C"

// ---- NCCL, bound at run time -------------------------------------------------------------------------
// The library does not link NCCL (a single GPU needs none of it). tsvm_shard_attach_nccl looks the few
// entry points up in the libnccl.so.2 the process already has (or can load) and keeps a communicator.
namespace {
typedef struct ncclComm *ncclComm_t;
struct ncclUniqueIdBytes { char internal[128]; };
enum { NCCL_INT32 = 2, NCCL_FLOAT32 = 7, NCCL_FLOAT64 = 8, NCCL_SUM = 0 };
struct NcclApi {
    int (*GetUniqueId)(ncclUniqueIdBytes *) = nullptr;
    int (*CommInitRank)(ncclComm_t *, int, ncclUniqueIdBytes, int) = nullptr;
    int (*CommDestroy)(ncclComm_t) = nullptr;
    int (*AllGather)(const void *, void *, size_t, int, ncclComm_t, cudaStream_t) = nullptr;
    int (*AllReduce)(const void *, void *, size_t, int, int, ncclComm_t, cudaStream_t) = nullptr;
    int (*GroupStart)() = nullptr;
    int (*GroupEnd)() = nullptr;
    const char *(*GetErrorString)(int) = nullptr;
    bool ok = false;
};
NcclApi &nccl_api() {
    static NcclApi api;
    static bool tried = false;
    if (tried) return api;
    tried = true;
    void *h = dlopen("libnccl.so.2", RTLD_NOW | RTLD_GLOBAL);
    if (!h) h = dlopen("libnccl.so", RTLD_NOW | RTLD_GLOBAL);
    if (!h) return api;
    api.GetUniqueId = (decltype(api.GetUniqueId)) dlsym(h, "ncclGetUniqueId");
    api.CommInitRank = (decltype(api.CommInitRank)) dlsym(h, "ncclCommInitRank");
    api.CommDestroy = (decltype(api.CommDestroy)) dlsym(h, "ncclCommDestroy");
    api.AllGather = (decltype(api.AllGather)) dlsym(h, "ncclAllGather");
    api.AllReduce = (decltype(api.AllReduce)) dlsym(h, "ncclAllReduce");
    api.GroupStart = (decltype(api.GroupStart)) dlsym(h, "ncclGroupStart");
    api.GroupEnd = (decltype(api.GroupEnd)) dlsym(h, "ncclGroupEnd");
    api.GetErrorString = (decltype(api.GetErrorString)) dlsym(h, "ncclGetErrorString");
    api.ok = api.GetUniqueId && api.CommInitRank && api.CommDestroy && api.AllGather && api.AllReduce &&
             api.GroupStart && api.GroupEnd && api.GetErrorString;
    return api;
}
}  // namespace
#define TSVM_NCCL(expr)                                                                                  \
    do {                                                                                                 \
        const int r__ = (expr);                                                                          \
        if (r__ != 0) {                                                                                  \
            tsvm::set_error("%s failed: %s", #expr, nccl_api().GetErrorString(r__));                     \
            return TSVM_ERR_CUDA;                                                                        \
        }                                                                                                \
    } while (0)

// Per-rank state of the column-sharded solver. The caller owns the exchange buffers (they are the operands of
// its collectives): cand_f/cand_id [lists * ws], all_f/all_id [world * lists * ws], crow [ws * (dp + 4)] floats,
// cstate [ws * 3] doubles.
struct tsvm_shard {
    tsvm_km *km = nullptr;
    int kind = 0, ws = 0, q = 0, n_local = 0, n_total = 0, lo = 0, hi = 0, world = 1, d = 0, dp = 0;
    const int *y = nullptr;
    double *alpha = nullptr, *f = nullptr;
    double eps = 0, Cp = 0, Cn = 0;
    long long ld = 0;
    cudaStream_t st = nullptr, st2 = nullptr;
    ncclComm_t comm = nullptr;       // set by tsvm_shard_attach_nccl (not owned): the library then runs the exchange steps itself
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_blk = nullptr;
    // timing events of the queued iterations: kernel-row launch (first stream), block + local solver (second)
    struct StepEvents { cudaEvent_t r0 = nullptr, r1 = nullptr, b0 = nullptr, b1 = nullptr; };
    StepEvents evs[MAX_QUEUED];
    int queued = 0;                  // iterations enqueued since the last read of the device's verdict
    SolverCtl *ctl = nullptr, *ctl_host = nullptr;   // termination rules applied on the device (solver_status_kernel)
    double t_rows = 0, t_loc = 0;    // ms
    // exchange buffers (caller's)
    double *cand_f = nullptr, *all_f = nullptr, *cstate = nullptr;
    int *cand_id = nullptr, *all_id = nullptr;
    float *crow = nullptr;
    // own buffers
    int *ids = nullptr, *y_ws = nullptr;
    float *rows = nullptr, *kww = nullptr, *m_hi = nullptr, *m_lo = nullptr, *m_sd = nullptr, *m_unscale = nullptr,
          *m_diag = nullptr;
    double *f_ws = nullptr, *a_ws = nullptr, *alpha_diff = nullptr, *diff = nullptr, *grp_f = nullptr;
    int *grp_id = nullptr;
    unsigned char *in_ws = nullptr;
    tsvm_ws *sel = nullptr;
    size_t row_bytes = 0;
    long long iter = 0, local_iter = 0, rows_made = 0, launches0 = 0;
    int local_max_iter = 0, n_new = 0, slot0 = 0, phase = 0;
    double diff0 = 0;
    bool done = false;
    std::chrono::steady_clock::time_point t_begin;

    ~tsvm_shard() {
        pool_free_many({ids, y_ws, rows, kww, m_hi, m_lo, m_sd, m_unscale, m_diag, f_ws, a_ws, alpha_diff, diff, grp_f,
                        grp_id, in_ws, ctl});
        tsvm_ws_destroy(sel);
        if (ctl_host) pinned_free(ctl_host);
        for (auto e : {ev_fork, ev_join, ev_blk}) if (e) cudaEventDestroy(e);
        for (auto &E : evs)
            for (auto e : {E.r0, E.r1, E.b0, E.b1}) if (e) cudaEventDestroy(e);
        if (st2) cudaStreamDestroy(st2);
    }

    tsvm_status init() {
        TSVM_REQUIRE(!km->from_csr && km_pair_engine(km, st), "shard solver: needs dense data on the CTA-pair tensor engine "
                                             "(more than 32 features)");
        km->launched(st);
        km->streams_mixed = true;        // (this solver's two streams; its calls do not note their work on the matrix one by one)
        row_bytes = km_plane_row_bytes(km);
        const size_t plane_words = (row_bytes * (size_t) ws + 3) / 4;
        TSVM_TRY(dev_alloc(&ids, (size_t) ws));
        TSVM_TRY(dev_alloc(&y_ws, (size_t) ws));
        TSVM_TRY(dev_alloc(&rows, (size_t) ws * ld));
        TSVM_TRY(dev_alloc(&kww, (size_t) ws * ws));
        TSVM_TRY(dev_alloc(&m_hi, plane_words));
        TSVM_TRY(dev_alloc(&m_lo, plane_words));
        TSVM_TRY(dev_alloc(&m_sd, (size_t) ws));
        TSVM_TRY(dev_alloc(&m_unscale, (size_t) ws));
        TSVM_TRY(dev_alloc(&m_diag, (size_t) ws));
        TSVM_TRY(dev_alloc(&f_ws, (size_t) ws));
        TSVM_TRY(dev_alloc(&a_ws, (size_t) ws));
        TSVM_TRY(dev_alloc(&alpha_diff, (size_t) ws));
        TSVM_TRY(dev_alloc(&diff, 4));
        TSVM_TRY(dev_alloc(&grp_f, (size_t) world * MAX_LISTS * ws));
        TSVM_TRY(dev_alloc(&grp_id, (size_t) world * MAX_LISTS * ws));
        TSVM_TRY(dev_alloc(&in_ws, (size_t) n_local));
        TSVM_CUDA(cudaMemsetAsync(in_ws, 0, (size_t) n_local, st));
        TSVM_TRY(ws_alloc(n_local, ws, &sel));
        TSVM_TRY(clear_select_state(sel, st));
        TSVM_TRY(dev_alloc(&ctl, 1));
        TSVM_TRY(pinned_alloc((void **) &ctl_host, sizeof(SolverCtl)));
        memset(ctl_host, 0, sizeof(SolverCtl));
        ctl_host->prev = ctl_host->last = ctl_host->second_last = INFINITY;     // csmosolver.cpp:51-57
        TSVM_CUDA(cudaMemcpyAsync(ctl, ctl_host, sizeof(SolverCtl), cudaMemcpyHostToDevice, st));
        TSVM_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
        TSVM_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
        TSVM_CUDA(cudaEventCreateWithFlags(&ev_blk, cudaEventDisableTiming));
        int lo_prio = 0, hi_prio = 0;
        TSVM_CUDA(cudaDeviceGetStreamPriorityRange(&lo_prio, &hi_prio));
        TSVM_CUDA(cudaStreamCreateWithPriority(&st2, cudaStreamNonBlocking, hi_prio));
        local_max_iter = ws > INT_MAX / 100 ? INT_MAX : (100 * ws > 100000 ? 100 * ws : 100000);
        return TSVM_OK;
    }

    // phase A: rotate the working set, then this rank's candidate lists (global ids) into cand_f / cand_id
    tsvm_status candidates(int *lists_out, int *want_out) {
        TSVM_REQUIRE(phase == 0, "shard solver: phases out of order (candidates)");
        const int lists = kind == TSVM_SOLVER_C ? 2 : 4;
        const long long it = iter + queued;         // the iteration being enqueued
        n_new = it == 0 ? ws : q;
        slot0 = it == 0 ? 0 : q;
        if (it > 0) {
            TSVM_LAUNCH(shard_shift_kernel, 1, 1024, 0, st, ids, q, lo, hi, in_ws, m_sd, m_unscale, m_diag);
            TSVM_CUDA(cudaMemcpyAsync(m_hi, (char *) m_hi + (size_t) q * row_bytes, (size_t) q * row_bytes,
                                      cudaMemcpyDeviceToDevice, st));
            TSVM_CUDA(cudaMemcpyAsync(m_lo, (char *) m_lo + (size_t) q * row_bytes, (size_t) q * row_bytes,
                                      cudaMemcpyDeviceToDevice, st));
        }
        // the best n_new of every list, sorted: the merge of the gathered sorted runs needs no sort
        TSVM_TRY(launch_select(sel, kind, n_local, f, alpha, y, it == 0 ? nullptr : in_ws, Cp, Cn, n_new, lo, cand_f, cand_id,
                               nullptr, &ctl->stop, st));
        *lists_out = lists;
        *want_out = n_new;
        phase = 1;
        return TSVM_OK;
    }

    // phase B: the same merge on every rank over the gathered lists, then this rank's contributions
    tsvm_status select() {
        TSVM_REQUIRE(phase == 1, "shard solver: phases out of order (select)");
        const int lists = kind == TSVM_SOLVER_C ? 2 : 4;
        const double *mf = all_f;
        const int *mi = all_id;
        if (world > 1) {
            TSVM_LAUNCH(shard_regroup_kernel, ceil_div(world * lists * n_new, 256), 256, 0, st, all_f, all_id, world,
                        lists, n_new, grp_f, grp_id);
            mf = grp_f; mi = grp_id;
        }
        TSVM_TRY(tsvm_ws_merge_sorted(sel, kind, mf, mi, world * n_new, n_new, n_new, ids + slot0, st));
        TSVM_LAUNCH(shard_contrib_kernel, n_new + 4, 256, 0, st, ids, slot0, n_new, ws, lo, hi, km->X, km->ldx, d, dp,
                    km->self_dot, km->diag, y, f, alpha, crow, cstate);
        phase = 2;
        return TSVM_OK;
    }

    // phase C: everything after the exchange, enqueued without waiting. The last launch applies the
    // termination rules on the device (solver_status_kernel); once it has set the stop word, the selection and
    // the local solver of any iteration queued behind it do nothing - the local solver leaves a zero step, so
    // the f updates subtract zero and the scatter writes back the alphas it read.
    tsvm_status enqueue_tail() {
        TSVM_REQUIRE(phase == 2, "shard solver: phases out of order (iterate)");
        TSVM_REQUIRE(queued < MAX_QUEUED, "shard solver: too many iterations queued");
        const long long it = iter + queued;
        const int first_half_phys = (int) (it & 1);
        StepEvents &E = evs[queued];
        if (!E.r0) for (auto e : {&E.r0, &E.r1, &E.b0, &E.b1}) TSVM_CUDA(cudaEventCreate(e));
        TSVM_LAUNCH(shard_unpack_kernel, ceil_div(ws, 256), 256, 0, st, crow, slot0, n_new, dp, ws, cstate, m_sd, m_diag,
                    y_ws, f_ws, a_ws);
        TSVM_TRY(km_stage_rows_features(km, crow, dp + 4, m_sd + slot0, n_new, st));
        TSVM_CUDA(cudaMemcpyAsync((char *) m_hi + (size_t) slot0 * row_bytes, km->Whi, (size_t) n_new * row_bytes,
                                  cudaMemcpyDeviceToDevice, st));
        TSVM_CUDA(cudaMemcpyAsync((char *) m_lo + (size_t) slot0 * row_bytes, km->Wlo, (size_t) n_new * row_bytes,
                                  cudaMemcpyDeviceToDevice, st));
        TSVM_CUDA(cudaMemcpyAsync(m_unscale + slot0, km->w_unscale, sizeof(float) * n_new, cudaMemcpyDeviceToDevice, st));
        TSVM_CUDA(cudaEventRecord(ev_fork, st));
        // second stream: the whole ws x ws block from the members' planes (every rank computes the same
        // values the owners' row buffers hold), then the local solver, replicated
        TSVM_CUDA(cudaStreamWaitEvent(st2, ev_fork, 0));
        const InstancePlanes members{m_hi, m_lo, m_sd, m_unscale, ws};
        const RowPlanes member_rows{m_hi, m_lo, m_sd, m_unscale};
        TSVM_CUDA(cudaEventRecord(E.b0, st2));
        TSVM_TRY(km_rows_planes_on(km, members, member_rows, ws, kww, ws, st2));
        // The kernel-row launch below leaves one SM pair free; started first it would leave the block's eight
        // pairs that one pair to run on, and the local solver - the longer of the two paths once the rows are
        // split - would start late. With iterations queued nothing else orders the two, so the first stream waits
        // for the block.
        TSVM_CUDA(cudaEventRecord(ev_blk, st2));
        TSVM_TRY(launch_local_smo(kind, ws, kww, m_diag, y_ws, f_ws, a_ws, alpha_diff, Cp, Cn, eps, local_max_iter, diff,
                                  nullptr, nullptr, st2, &ctl->stop));
        TSVM_CUDA(cudaEventRecord(E.b1, st2));
        if (it > 0)        // the old half's rows are in the buffer already
            TSVM_TRY(launch_update_f(f, n_local, alpha_diff, q, first_half_phys, rows, ld, 0, 0, q, nullptr, st2));
        TSVM_CUDA(cudaEventRecord(ev_join, st2));
        // first stream: the new rows against this rank's columns
        float *new_rows = rows + (size_t) (it == 0 ? 0 : (1 - first_half_phys) * q) * ld;
        km->reserve_clusters = 1;
        TSVM_CUDA(cudaStreamWaitEvent(st, ev_blk, 0));
        TSVM_CUDA(cudaEventRecord(E.r0, st));
        const tsvm_status rs = km_rows_staged(km, n_new, new_rows, ld, st);
        km->reserve_clusters = 0;
        TSVM_TRY(rs);
        TSVM_CUDA(cudaEventRecord(E.r1, st));
        TSVM_CUDA(cudaStreamWaitEvent(st, ev_join, 0));
        TSVM_TRY(launch_update_f(f, n_local, alpha_diff, q, first_half_phys, rows, ld, it == 0 ? 0 : q, it == 0 ? 0 : q, ws, nullptr, st));
        TSVM_LAUNCH(shard_scatter_kernel, ceil_div(ws, 256), 256, 0, st, ids, ws, lo, hi, a_ws, alpha);
        StatusArgs status;
        status.c = ctl; status.diff = diff; status.got = sel->count; status.wanted = n_new; status.eps = eps;
        status.engine_status = km->status_dev;
        TSVM_LAUNCH(solver_status_kernel, 1, 32, 0, st, status);
        ++queued;
        phase = 0;
        return TSVM_OK;
    }

    // Waits for the queued iterations and takes over what the device decided (fewer than queued may have run).
    tsvm_status collect() {
        if (queued == 0) return TSVM_OK;
        TSVM_CUDA(cudaMemcpyAsync(ctl_host, ctl, sizeof(SolverCtl), cudaMemcpyDeviceToHost, st));
        TSVM_CUDA(cudaStreamSynchronize(st));
        const SolverCtl &c = *ctl_host;
        const int was_queued = queued;
        queued = 0;
        if (c.engine_status != 0) {
            set_error("dense kernel-row engine reported status %d (a bounded wait ran out)", c.engine_status);
            return TSVM_ERR_DEVICE;
        }
        const int ran = (int) (c.iter - iter);
        for (int j = 0; j < ran && j < was_queued; ++j) {
            float ms_ev = 0;
            cudaEventElapsedTime(&ms_ev, evs[j].r0, evs[j].r1); t_rows += ms_ev;
            cudaEventElapsedTime(&ms_ev, evs[j].b0, evs[j].b1); t_loc += ms_ev;
            rows_made += iter + j == 0 ? ws : q;
        }
        iter = c.iter;
        local_iter = c.local_iter;
        diff0 = c.diff0;
        done = c.done != 0;
        if (c.short_wanted > 0) {
            set_error("working-set selection found %d eligible instances for %d slots (is a class weight or C zero?)",
                      c.short_got, c.short_wanted);
            return TSVM_ERR_INVALID;
        }
        return TSVM_OK;
    }

    tsvm_status iterate() {
        TSVM_TRY(enqueue_tail());
        return collect();
    }

    // One whole outer iteration with the exchange steps enqueued on the solver's stream by the library
    // (needs a communicator): no host work between the phases.
    tsvm_status step() {
        TSVM_REQUIRE(comm || world == 1, "shard solver: tsvm_shard_step needs tsvm_shard_attach_nccl first");
        int lists = 0, want = 0;
        TSVM_TRY(candidates(&lists, &want));
        const size_t m = (size_t) lists * want;
        if (world > 1) {
            NcclApi &nc = nccl_api();
            TSVM_NCCL(nc.GroupStart());
            TSVM_NCCL(nc.AllGather(cand_f, all_f, m, NCCL_FLOAT64, comm, st));
            TSVM_NCCL(nc.AllGather(cand_id, all_id, m, NCCL_INT32, comm, st));
            TSVM_NCCL(nc.GroupEnd());
        } else {
            TSVM_CUDA(cudaMemcpyAsync(all_f, cand_f, m * sizeof(double), cudaMemcpyDeviceToDevice, st));
            TSVM_CUDA(cudaMemcpyAsync(all_id, cand_id, m * sizeof(int), cudaMemcpyDeviceToDevice, st));
        }
        TSVM_TRY(select());
        if (world > 1) {
            NcclApi &nc = nccl_api();
            TSVM_NCCL(nc.GroupStart());
            TSVM_NCCL(nc.AllReduce(crow, crow, (size_t) n_new * (dp + 4), NCCL_FLOAT32, NCCL_SUM, comm, st));
            TSVM_NCCL(nc.AllReduce(cstate, cstate, (size_t) ws * 3, NCCL_FLOAT64, NCCL_SUM, comm, st));
            TSVM_NCCL(nc.GroupEnd());
        }
        return enqueue_tail();
    }

    // Up to n_iters whole iterations, queued sync_every() at a time between reads of the device's verdict.
    tsvm_status run(int n_iters) {
        for (long long end = iter + n_iters; iter < end && !done;) {
            long long k = end - iter;
            if (k > sync_every()) k = sync_every();
            if (iter == 0) k = 1;                   // the first iteration is read back on its own
            for (int j = 0; j < (int) k; ++j) {
                const tsvm_status s = step();
                if (s != TSVM_OK) { collect(); return s; }
            }
            TSVM_TRY(collect());
        }
        return TSVM_OK;
    }
};

extern "C" {

int tsvm_nccl_unique_id(void *id128) {
    NcclApi &nc = nccl_api();
    if (!nc.ok || !id128) { tsvm::set_error("NCCL is not available in this process (libnccl.so.2 not found)"); return TSVM_ERR_INVALID; }
    ncclUniqueIdBytes id;
    const int r = nc.GetUniqueId(&id);
    if (r != 0) { tsvm::set_error("ncclGetUniqueId failed: %s", nc.GetErrorString(r)); return TSVM_ERR_CUDA; }
    memcpy(id128, &id, sizeof(id));
    return TSVM_OK;
}

tsvm_status tsvm_nccl_comm_create(const void *id128, int rank, int world, void **comm_out) {
    TSVM_REQUIRE(id128 && comm_out && world >= 1 && rank >= 0 && rank < world, "nccl_comm_create: bad arguments");
    NcclApi &nc = nccl_api();
    TSVM_REQUIRE(nc.ok, "NCCL is not available in this process (libnccl.so.2 not found)");
    ncclUniqueIdBytes id;
    memcpy(&id, id128, sizeof(id));
    ncclComm_t c = nullptr;
    TSVM_NCCL(nc.CommInitRank(&c, world, id, rank));
    *comm_out = c;
    return TSVM_OK;
}

void tsvm_nccl_comm_destroy(void *comm) {
    if (comm && nccl_api().ok) nccl_api().CommDestroy((ncclComm_t) comm);
}

tsvm_status tsvm_shard_attach_nccl(tsvm_shard *S, void *comm) {
    TSVM_REQUIRE(S && comm, "shard_attach_nccl: null argument");
    S->comm = (ncclComm_t) comm;
    return TSVM_OK;
}

tsvm_status tsvm_shard_step(tsvm_shard *S, int *done_host) {
    TSVM_REQUIRE(S && done_host, "shard_step: null argument");
    TSVM_TRY(S->run(1));
    *done_host = S->done ? 1 : 0;
    return TSVM_OK;
}

tsvm_status tsvm_shard_run(tsvm_shard *S, int n_iters, int *done_host) {
    TSVM_REQUIRE(S && n_iters > 0, "shard_run: bad arguments");
    TSVM_TRY(S->run(n_iters));
    if (done_host) *done_host = S->done ? 1 : 0;
    return TSVM_OK;
}

tsvm_status tsvm_shard_create(tsvm_km *km_local, int solver_kind, const int *y_dev, double *alpha_dev, double *f_dev,
                              int n_total, int lo, double eps, double Cp, double Cn, int ws_size, int world,
                              double *cand_f_dev, int *cand_id_dev, double *all_f_dev, int *all_id_dev,
                              float *rows_contrib_dev, double *state_contrib_dev, void *stream, tsvm_shard **out) {
    TSVM_REQUIRE(out && km_local && y_dev && alpha_dev && f_dev && cand_f_dev && cand_id_dev && all_f_dev &&
                 all_id_dev && rows_contrib_dev && state_contrib_dev, "shard_create: null argument");
    TSVM_REQUIRE(solver_kind >= 0 && solver_kind <= 2, "shard_create: unknown solver %d", solver_kind);
    TSVM_REQUIRE(world >= 1 && lo >= 0 && lo + km_local->n <= n_total, "shard_create: bad ownership range");
    TSVM_REQUIRE(ws_size >= 2 && ws_size <= 1024 && ws_size <= n_total && (ws_size & (ws_size - 1)) == 0 &&
                 (long long) world * ws_size <= MERGE_MAX_LEN,
                 "shard_create: working-set size %d must be a power of two in [2, min(n, 1024)] and world * ws <= %d",
                 ws_size, MERGE_MAX_LEN);
    *out = nullptr;
    tsvm_shard *S = new tsvm_shard;
    S->km = km_local; S->kind = solver_kind; S->y = y_dev; S->alpha = alpha_dev; S->f = f_dev;
    S->eps = eps; S->Cp = Cp; S->Cn = Cn; S->ws = ws_size; S->q = ws_size / 2;
    S->n_local = km_local->n; S->n_total = n_total; S->lo = lo; S->hi = lo + km_local->n; S->world = world;
    S->d = km_local->d; S->dp = (km_local->d + 3) & ~3;
    S->ld = ((long long) km_local->n + 3) & ~3ll;
    S->st = (cudaStream_t) stream;
    S->cand_f = cand_f_dev; S->cand_id = cand_id_dev; S->all_f = all_f_dev; S->all_id = all_id_dev;
    S->crow = rows_contrib_dev; S->cstate = state_contrib_dev;
    S->launches0 = launch_count();
    S->t_begin = std::chrono::steady_clock::now();
    tsvm_status s = S->init();
    if (s != TSVM_OK) { delete S; return s; }
    *out = S;
    return TSVM_OK;
}

tsvm_status tsvm_shard_candidates(tsvm_shard *S, int *lists_host, int *want_host) {
    TSVM_REQUIRE(S && lists_host && want_host, "shard_candidates: null argument");
    return S->candidates(lists_host, want_host);
}

tsvm_status tsvm_shard_select(tsvm_shard *S, int *n_new_host) {
    TSVM_REQUIRE(S && n_new_host, "shard_select: null argument");
    TSVM_TRY(S->select());
    *n_new_host = S->n_new;
    return TSVM_OK;
}

tsvm_status tsvm_shard_iterate(tsvm_shard *S, int *done_host) {
    TSVM_REQUIRE(S && done_host, "shard_iterate: null argument");
    TSVM_TRY(S->iterate());
    *done_host = S->done ? 1 : 0;
    return TSVM_OK;
}

tsvm_status tsvm_shard_get_stats(const tsvm_shard *S, tsvm_solve_stats *out) {
    TSVM_REQUIRE(S && out, "shard_get_stats: null argument");
    memset(out, 0, sizeof(*out));
    out->outer_iters = S->iter;
    out->local_iters = S->local_iter;
    out->final_diff = S->diff0;
    out->objective = NAN;
    out->seconds_rows = S->t_rows * 1e-3;
    out->seconds_local = S->t_loc * 1e-3;       // ws x ws block + local solver, on the second stream
    out->seconds_total = std::chrono::duration<double>(std::chrono::steady_clock::now() - S->t_begin).count();
    out->kernel_rows = S->rows_made;
    out->gpu_launches = launch_count() - S->launches0;
    return TSVM_OK;
}

void tsvm_shard_destroy(tsvm_shard *S) { delete S; }

}  // extern "C"
