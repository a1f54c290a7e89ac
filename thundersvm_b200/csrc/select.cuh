// Working-set selection.
//
// The reference sorts all n f-values every outer iteration (src/thundersvm/kernel/smo_kernel.cu:312-315) and then walks
// the sorted ids from both ends on the host (src/thundersvm/solver/csmosolver.cpp:123-165). Only the first `want`
// eligible instances of every walk can ever be taken, so the device keeps, per walk ("list"), the `want` smallest
// 96-bit keys (f-order, id) among the eligible instances:
//   C-SMO : list 0 = I_up ascending (f, id);      list 1 = I_low descending (f, id)
//   nu-SMO: lists 0/1 = I_up for y>0 / y<0;       lists 2/3 = I_low for y>0 / y<0
// and merges them in the reference's alternating order.
//
// What bounds it: latency. The data is a few megabytes at most; what costs is every pass over it that has to wait for
// the pass before. select_kernel therefore makes ONE pass over all instances and crosses the grid twice:
//   1. every block finds the same pivot of every list from the same sample of the instances (radix select over the
//      sample in shared memory; no communication)
//   2. one sweep collects the instances up to the pivot: a few hundred more than wanted          -- grid barrier --
//   3. the candidates' ranks are counted (each against all others, over all blocks): the sorted lists -- last block --
//   4. one block merges the lists
// A pivot that was too small or too large - the sample was not typical - is replaced by an exact radix select over all
// instances (exact_pivots: 12-bit digits, one sweep and one grid barrier each). Exact and deterministic either way.
//
// (Measured: see select_grid.)
#pragma once
#include "common.cuh"
#include <cooperative_groups.h>

namespace tsvm {

constexpr int RADIX_BITS = 12, RADIX_BINS = 1 << RADIX_BITS, RADIX_PASSES = 8, MAX_LISTS = 4;
typedef unsigned __int128 key96_t;

struct SelectState {            // one per list, lives in device memory
    unsigned long long prefix_hi;   // exact_pivots: bits 95..32 of the threshold key found so far
    unsigned int prefix_lo;         // bits 31..0
    int k_rem;                      // rank still to resolve inside the current prefix
    int take_all;                   // fewer eligible instances than wanted: take every one
    int count;                      // candidates collected (zero between calls)
    int resolved;                   // the threshold is final: later radix passes skip this list
};

__device__ __forceinline__ int list_count(int solver_kind) { return solver_kind == TSVM_SOLVER_C ? 2 : 4; }

// Is instance (a, y) eligible for list l?
__device__ __forceinline__ bool in_list(int solver_kind, int l, double a, int y, double Cp, double Cn) {
    if (solver_kind == TSVM_SOLVER_C) return l == 0 ? in_I_up(a, y, Cp, Cn) : in_I_low(a, y, Cp, Cn);
    const bool pos = (l & 1) == 0;
    if (pos != (y > 0)) return false;
    return l < 2 ? in_I_up(a, y, Cp, Cn) : in_I_low(a, y, Cp, Cn);
}
// All lists at once, bit l = list l
__device__ __forceinline__ unsigned lists_of(int solver_kind, double a, int y, double Cp, double Cn) {
    const unsigned up = in_I_up(a, y, Cp, Cn) ? 1u : 0u, low = in_I_low(a, y, Cp, Cn) ? 1u : 0u;
    if (solver_kind == TSVM_SOLVER_C) return up | low << 1;
    return (up | low << 2) << (y > 0 ? 0 : 1);
}
__device__ __forceinline__ bool list_ascending(int solver_kind, int l) {
    return solver_kind == TSVM_SOLVER_C ? l == 0 : l < 2;
}
__device__ __forceinline__ key96_t make_key(bool asc, double f, unsigned id) {
    unsigned long long h = ordered_key(f);
    if (!asc) { h = ~h; id = ~id; }
    return ((key96_t) h << 32) | id;
}

__device__ __forceinline__ bool key_less(unsigned long long ah, unsigned al, unsigned long long bh, unsigned bl) {
    return ah < bh || (ah == bh && al < bl);
}

// ---- merge: sort every candidate list, keep its first `want`, then the reference's alternating
// walk with "already taken" checks (csmosolver.cpp:123-165 / nusmosolver.cpp:48-118). ------------
constexpr int MERGE_THREADS = 1024, MERGE_MAX_LEN = 8192, MERGE_MAX_WANT = 1024, HASH_SLOTS = 4096;
constexpr int MERGE_JOINT_MAX = 2048;          // longest lists that merge_lists sorts side by side

// The reference's alternating walk over the sorted lists: top_id [lists][MERGE_MAX_WANT] holds the first top_len[l] ids of
// every list, last_fkey[l] the f-order key of the last of them, partner [lists][MERGE_MAX_WANT] is -1 everywhere. One
// block of MERGE_THREADS threads, after a barrier.
__device__ void walk_lists(int lists, int want, const int *top_id, short *partner, int *hash_id, short *hash_pos,
                           const int *top_len, const unsigned long long *last_fkey, int *__restrict__ out_ids,
                           int *__restrict__ out_count) {
    const int tid = threadIdx.x;
    // An instance sits in an "up" list and in the paired "low" list only if the up list's largest f is not
    // below the low list's smallest f. For large problems that never happens: no instance is then met twice,
    // the reference's alternating walk takes entry p of every list in round p, and the output position of
    // every entry follows from the list lengths alone.
    const int half = lists / 2;
    bool disjoint = true;
    for (int u = 0; u < half; ++u)
        if (top_len[u] > 0 && top_len[u + half] > 0 && !(last_fkey[u] < last_fkey[u + half])) disjoint = false;
    if (disjoint) {
        int total = 0;
        for (int l = 0; l < lists; ++l) total += top_len[l];
        const int got = total < want ? total : want;
        for (int e = tid; e < lists * want; e += MERGE_THREADS) {
            const int l = e / want, p = e - l * want;
            if (p >= top_len[l]) continue;
            int pos = 0;
            for (int o = 0; o < lists; ++o) pos += (top_len[o] < p ? top_len[o] : p) + ((o < l && top_len[o] > p) ? 1 : 0);
            if (pos < want) out_ids[pos] = top_id[l * MERGE_MAX_WANT + p];
        }
        for (int r = got + tid; r < want; r += MERGE_THREADS) out_ids[r] = -1;
        if (tid == 0 && out_count) *out_count = got;
        return;
    }

    // partner positions: an instance can sit in an "up" list and in the "low" list of the same
    // class. up list u pairs with low list u + lists/2.
    for (int u = 0; u < half; ++u) {
        const int lw = u + half;
        for (int s = tid; s < HASH_SLOTS; s += MERGE_THREADS) hash_id[s] = -1;
        __syncthreads();
        for (int e = tid; e < top_len[lw]; e += MERGE_THREADS) {
            const int id = top_id[lw * MERGE_MAX_WANT + e];
            unsigned s = ((unsigned) id * 2654435761u) >> 20;
            for (;;) {
                const int old = atomicCAS(&hash_id[s], -1, id);
                if (old == -1) { hash_pos[s] = (short) e; break; }
                s = (s + 1) & (HASH_SLOTS - 1);
            }
        }
        __syncthreads();
        for (int e = tid; e < top_len[u]; e += MERGE_THREADS) {
            const int id = top_id[u * MERGE_MAX_WANT + e];
            unsigned s = ((unsigned) id * 2654435761u) >> 20;
            for (;;) {
                const int cur = hash_id[s];
                if (cur == -1) break;
                if (cur == id) {
                    const short p = hash_pos[s];
                    partner[u * MERGE_MAX_WANT + e] = p;
                    partner[lw * MERGE_MAX_WANT + p] = (short) e;
                    break;
                }
                s = (s + 1) & (HASH_SLOTS - 1);
            }
        }
        __syncthreads();
    }

    // The walk takes the lists in turn, one entry each per round, and steps over an entry whose instance the partner
    // list has taken. Entry p of a list is reached in round t(p) = p - (entries stepped over before p); the up list,
    // whose turn comes first in a round, loses a shared instance if the low list reaches it in an earlier round, and
    // the low list loses it otherwise. Every decision depends on earlier rounds only, so repeating "decide from t,
    // recompute t by a prefix sum" from t(p) = p settles on the walk's own outcome, in two or three rounds for the
    // usual case of two lists that run towards each other (one thread walking it took 40 us for 512 ids).
    static_assert(MERGE_MAX_WANT <= MERGE_THREADS, "one list entry per thread");
    short *when = reinterpret_cast<short *>(hash_id);                   // [lists][want]: t(p); the hash table is done with
    static_assert(MAX_LISTS * MERGE_MAX_WANT * sizeof(short) <= HASH_SLOTS * sizeof(int), "t(p) does not fit the hash table");
    __shared__ int step_over[MAX_LISTS][MERGE_THREADS / 32];
    __shared__ int n_taken[MAX_LISTS];
    const int lane = tid & 31, warp = tid >> 5;
    int t_own[MAX_LISTS];
    short mate[MAX_LISTS];
    unsigned stepped = 0;                       // bit l: this thread's entry of list l is stepped over
#pragma unroll
    for (int l = 0; l < MAX_LISTS; ++l) {
        t_own[l] = tid;
        mate[l] = l < lists && tid < top_len[l] ? partner[l * MERGE_MAX_WANT + tid] : (short) -1;
    }
    for (;;) {
        __syncthreads();                        // (first round: everyone is done with the hash table)
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l)
            if (l < lists) when[l * MERGE_MAX_WANT + tid] = (short) t_own[l];
        __syncthreads();
        unsigned over[MAX_LISTS];
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l) {
            bool skip = false;
            if (l < lists && mate[l] >= 0) {
                const int other = when[(l < half ? l + half : l - half) * MERGE_MAX_WANT + mate[l]];
                skip = l < half ? other < t_own[l] : other <= t_own[l];
            }
            over[l] = __ballot_sync(0xffffffffu, skip);
            if (lane == 0) step_over[l][warp] = __popc(over[l]);
        }
        __syncthreads();
        bool changed = false;
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l) {
            if (l >= lists) continue;
            int before = lane < warp ? step_over[l][lane] : 0;
            before = __reduce_add_sync(0xffffffffu, before) + __popc(over[l] & ((1u << lane) - 1));
            changed = changed || (tid < top_len[l] && t_own[l] != tid - before);
            t_own[l] = tid - before;
            stepped = (stepped & ~(1u << l)) | (((over[l] >> lane) & 1u) << l);
        }
        if (!__syncthreads_or(changed)) break;
    }
    if (tid < lists) {
        int sum = 0;
        for (int w = 0; w < MERGE_THREADS / 32; ++w) sum += step_over[tid][w];
        n_taken[tid] = top_len[tid] - sum;
    }
    __syncthreads();
    int total = 0;
    for (int l = 0; l < lists; ++l) total += n_taken[l];
    const int got = total < want ? total : want;
#pragma unroll
    for (int l = 0; l < MAX_LISTS; ++l) {
        if (l >= lists || tid >= top_len[l] || ((stepped >> l) & 1u)) continue;
        const int t = t_own[l];
        int pos = 0;
        for (int o = 0; o < lists; ++o) pos += (n_taken[o] < t ? n_taken[o] : t) + ((o < l && n_taken[o] > t) ? 1 : 0);
        if (pos < want) out_ids[pos] = top_id[l * MERGE_MAX_WANT + tid];
    }
    for (int r = got + tid; r < want; r += MERGE_THREADS) out_ids[r] = -1;
    if (tid == 0 && out_count) *out_count = got;
}

__device__ void merge_lists(int solver_kind, const double *__restrict__ cand_f, const int *__restrict__ cand_id, int len,
                            int want, int *__restrict__ out_ids, int *__restrict__ out_count, int seg_len,
                            unsigned char *smem) {
    const int lists = list_count(solver_kind);
    int P = 1;
    while (P < len) P <<= 1;
    // layout: sort keys (P x 12 B), then per list: top ids / partner positions
    unsigned long long *kh = reinterpret_cast<unsigned long long *>(smem);
    unsigned int *kl = reinterpret_cast<unsigned int *>(kh + P);
    int *top_id = reinterpret_cast<int *>(kl + P);                 // [lists][want]
    short *partner = reinterpret_cast<short *>(top_id + MAX_LISTS * MERGE_MAX_WANT);   // [lists][want]
    int *hash_id = reinterpret_cast<int *>(partner + MAX_LISTS * MERGE_MAX_WANT);      // [HASH_SLOTS]
    short *hash_pos = reinterpret_cast<short *>(hash_id + HASH_SLOTS);
    __shared__ int top_len[MAX_LISTS];
    __shared__ unsigned long long last_fkey[MAX_LISTS];
    __shared__ int real_total;
    const int tid = threadIdx.x;

    // Lists that are not made of sorted runs and fit the shared memory side by side are sorted together: every
    // step of the bitonic network handles all lists before its barrier (half the barriers for two lists).
    const bool joint = seg_len == 0 && P <= MERGE_JOINT_MAX;
    if (joint) {
        for (int l = 0; l < lists; ++l) {
            const bool asc = list_ascending(solver_kind, l);
            for (int e = tid; e < P; e += MERGE_THREADS) {
                unsigned long long h = ~0ull;
                unsigned lo = ~0u;
                if (e < len) {
                    const int id = __ldcg(cand_id + (size_t) l * len + e);
                    if (id >= 0) {
                        h = ordered_key(__ldcg(cand_f + (size_t) l * len + e));
                        lo = (unsigned) id;
                        if (!asc) { h = ~h; lo = ~lo; }
                    }
                }
                kh[(size_t) l * P + e] = h;
            }
        }
        // (kl follows all lists' kh)
        unsigned int *klj = reinterpret_cast<unsigned int *>(kh + (size_t) lists * P);
        for (int l = 0; l < lists; ++l) {
            const bool asc = list_ascending(solver_kind, l);
            for (int e = tid; e < P; e += MERGE_THREADS) {
                unsigned lo = ~0u;
                if (e < len) {
                    const int id = __ldcg(cand_id + (size_t) l * len + e);
                    if (id >= 0) lo = asc ? (unsigned) id : ~(unsigned) id;
                }
                klj[(size_t) l * P + e] = lo;
            }
        }
        __syncthreads();
        for (int k = 2; k <= P; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int w = tid; w < lists * (P >> 1); w += MERGE_THREADS) {
                    // comparison w of this step: list l, lower element e (bit j clear), partner e | j
                    const int l = w / (P >> 1), c = w - l * (P >> 1);
                    const int e = ((c & ~(j - 1)) << 1) | (c & (j - 1));
                    const int x = e | j;
                    unsigned long long *khl = kh + (size_t) l * P;
                    unsigned int *kll = klj + (size_t) l * P;
                    const bool up = (e & k) == 0;
                    if (key_less(khl[x], kll[x], khl[e], kll[e]) == up) {
                        unsigned long long th = khl[e]; khl[e] = khl[x]; khl[x] = th;
                        unsigned tl = kll[e]; kll[e] = kll[x]; kll[x] = tl;
                    }
                }
                __syncthreads();
            }
        int *top_id_j = reinterpret_cast<int *>(klj + (size_t) lists * P);
        top_id = top_id_j;
        partner = reinterpret_cast<short *>(top_id + MAX_LISTS * MERGE_MAX_WANT);
        hash_id = reinterpret_cast<int *>(partner + MAX_LISTS * MERGE_MAX_WANT);
        hash_pos = reinterpret_cast<short *>(hash_id + HASH_SLOTS);
        for (int l = 0; l < lists; ++l) {
            const bool asc = list_ascending(solver_kind, l);
            const unsigned long long *khl = kh + (size_t) l * P;
            const unsigned int *kll = klj + (size_t) l * P;
            for (int e = tid; e < want; e += MERGE_THREADS) {
                int id = -1;
                if (e < P && !(khl[e] == ~0ull && kll[e] == ~0u)) id = (int) (asc ? kll[e] : ~kll[e]);
                top_id[l * MERGE_MAX_WANT + e] = id;
                partner[l * MERGE_MAX_WANT + e] = -1;
            }
        }
        __syncthreads();
        if (tid < lists) {
            const int l = tid;
            const bool asc = list_ascending(solver_kind, l);
            const unsigned long long *khl = kh + (size_t) l * P;
            int c = want < P ? want : P;
            int lo = 0, hi = c;
            while (lo < hi) { int mid = (lo + hi) >> 1; if (top_id[l * MERGE_MAX_WANT + mid] >= 0) lo = mid + 1; else hi = mid; }
            top_len[l] = lo;
            last_fkey[l] = lo > 0 ? (asc ? khl[lo - 1] : ~khl[lo - 1]) : 0ull;
        }
        __syncthreads();
    }

    for (int l = 0; l < lists && !joint; ++l) {
        const bool asc = list_ascending(solver_kind, l);
        for (int e = tid; e < P; e += MERGE_THREADS) {
            unsigned long long h = ~0ull;
            unsigned lo = ~0u;
            if (e < len) {
                const int id = __ldcg(cand_id + (size_t) l * len + e);      // written by other blocks: from L2
                if (id >= 0) {
                    h = ordered_key(__ldcg(cand_f + (size_t) l * len + e));
                    lo = (unsigned) id;
                    if (!asc) { h = ~h; lo = ~lo; }
                    // keep real keys distinct from the padding key
                }
            }
            kh[e] = h; kl[e] = lo;
        }
        __syncthreads();
        if (seg_len > 0) {
            // The list is a sequence of sorted runs (one per rank, padding last): an entry's place in the merged
            // order is its place in its own run plus, for every other run, the number of smaller keys there
            // (binary search; keys are distinct because ids are). No sort, a few microseconds for 8 x 512.
            const int nseg = len / seg_len;
            for (int e = tid; e < want; e += MERGE_THREADS) {
                top_id[l * MERGE_MAX_WANT + e] = -1;
                partner[l * MERGE_MAX_WANT + e] = -1;
            }
            if (tid == 0) real_total = 0;
            __syncthreads();
            if (tid < nseg) {                       // real entries of run tid: first padding key
                int lo_i = 0, hi_i = seg_len;
                while (lo_i < hi_i) {
                    const int mid = (lo_i + hi_i) >> 1;
                    const int e = tid * seg_len + mid;
                    if (kh[e] == ~0ull && kl[e] == ~0u) hi_i = mid; else lo_i = mid + 1;
                }
                atomicAdd(&real_total, lo_i);
            }
            __syncthreads();
            const int keep = real_total < want ? real_total : want;
            for (int e = tid; e < len; e += MERGE_THREADS) {
                const unsigned long long h = kh[e];
                const unsigned lo = kl[e];
                if (h == ~0ull && lo == ~0u) continue;
                const int r = e / seg_len;
                int rank = e - r * seg_len;
                for (int r2 = 0; r2 < nseg && rank < want; ++r2) {
                    if (r2 == r) continue;
                    int lo_i = 0, hi_i = seg_len;            // number of keys in run r2 below (h, lo)
                    while (lo_i < hi_i) {
                        const int mid = (lo_i + hi_i) >> 1;
                        const int x = r2 * seg_len + mid;
                        if (key_less(kh[x], kl[x], h, lo)) lo_i = mid + 1; else hi_i = mid;
                    }
                    rank += lo_i;
                }
                if (rank < want) {
                    top_id[l * MERGE_MAX_WANT + rank] = (int) (asc ? lo : ~lo);
                    if (rank == keep - 1) last_fkey[l] = asc ? h : ~h;
                }
            }
            if (tid == 0) { top_len[l] = keep; if (keep == 0) last_fkey[l] = 0ull; }
            __syncthreads();
            continue;
        }
        for (int k = 2; k <= P; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int e = tid; e < P; e += MERGE_THREADS) {
                    const int x = e ^ j;
                    if (x > e) {
                        const bool up = (e & k) == 0;
                        const bool lt = key_less(kh[x], kl[x], kh[e], kl[e]);
                        if (lt == up) {
                            unsigned long long th = kh[e]; kh[e] = kh[x]; kh[x] = th;
                            unsigned tl = kl[e]; kl[e] = kl[x]; kl[x] = tl;
                        }
                    }
                }
                __syncthreads();
            }
        for (int e = tid; e < want; e += MERGE_THREADS) {
            int id = -1;
            if (e < P && !(kh[e] == ~0ull && kl[e] == ~0u)) id = (int) (asc ? kl[e] : ~kl[e]);
            top_id[l * MERGE_MAX_WANT + e] = id;
            partner[l * MERGE_MAX_WANT + e] = -1;
        }
        __syncthreads();
        if (tid == 0) {
            int c = want < P ? want : P;
            // entries are sorted, padding last: count the real ones
            int lo = 0, hi = c;
            while (lo < hi) { int mid = (lo + hi) >> 1; if (top_id[l * MERGE_MAX_WANT + mid] >= 0) lo = mid + 1; else hi = mid; }
            top_len[l] = lo;
            // f-order key of the last kept entry: the list's largest f (ascending) / smallest f (descending)
            last_fkey[l] = lo > 0 ? (asc ? kh[lo - 1] : ~kh[lo - 1]) : 0ull;
        }
        __syncthreads();
    }

    walk_lists(lists, want, top_id, partner, hash_id, hash_pos, top_len, last_fkey, out_ids, out_count);
}

__global__ void __launch_bounds__(MERGE_THREADS)
select_merge_kernel(int solver_kind, const double *__restrict__ cand_f, const int *__restrict__ cand_id, int len,
                    int want, int *__restrict__ out_ids, int *__restrict__ out_count, int seg_len) {
    extern __shared__ unsigned char smem[];
    merge_lists(solver_kind, cand_f, cand_id, len, want, out_ids, out_count, seg_len, smem);
}

// Sorts a candidate list by its list key (padding, id -1, last): one block per list, bitonic in shared
// memory. The runs of several ranks can then be merged by rank computation instead of a sort.
__device__ void sort_list(int solver_kind, int l, const double *cand_f, const int *cand_id, int len, double *out_f,
                          int *out_id, int out_len, unsigned char *smem) {
    const int tid = threadIdx.x;
    int P = 1;
    while (P < len) P <<= 1;
    unsigned long long *kh = reinterpret_cast<unsigned long long *>(smem);
    unsigned int *kl = reinterpret_cast<unsigned int *>(kh + P);
    double *fv = reinterpret_cast<double *>(kl + P + (P & 1));          // the f values travel with their keys
    const bool asc = list_ascending(solver_kind, l);
    for (int e = tid; e < P; e += MERGE_THREADS) {
        unsigned long long h = ~0ull;
        unsigned lo = ~0u;
        double v = 0.0;
        if (e < len) {
            const int id = __ldcg(cand_id + (size_t) l * len + e);
            if (id >= 0) {
                v = __ldcg(cand_f + (size_t) l * len + e);
                h = ordered_key(v);
                lo = (unsigned) id;
                if (!asc) { h = ~h; lo = ~lo; }
            }
        }
        kh[e] = h; kl[e] = lo; fv[e] = v;
    }
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int e = tid; e < P; e += MERGE_THREADS) {
                const int x = e ^ j;
                if (x > e) {
                    const bool up = (e & k) == 0;
                    if (key_less(kh[x], kl[x], kh[e], kl[e]) == up) {
                        unsigned long long th = kh[e]; kh[e] = kh[x]; kh[x] = th;
                        unsigned tl = kl[e]; kl[e] = kl[x]; kl[x] = tl;
                        double tv = fv[e]; fv[e] = fv[x]; fv[x] = tv;
                    }
                }
            }
            __syncthreads();
        }
    // the first out_len entries of the sorted list (out_len <= len; the output may be the input)
    for (int e = tid; e < out_len; e += MERGE_THREADS) {
        const bool pad = kh[e] == ~0ull && kl[e] == ~0u;
        out_f[(size_t) l * out_len + e] = pad ? 0.0 : fv[e];
        out_id[(size_t) l * out_len + e] = pad ? -1 : (int) (asc ? kl[e] : ~kl[e]);
    }
}

__global__ void __launch_bounds__(MERGE_THREADS)
select_sort_candidates_kernel(int solver_kind, const double *cand_f, const int *cand_id, int len, double *out_f,
                              int *out_id, int out_len) {
    extern __shared__ unsigned char smem[];
    sort_list(solver_kind, blockIdx.x, cand_f, cand_id, len, out_f, out_id, out_len, smem);
}

static size_t merge_smem_bytes(int len) {
    int P = 1;
    while (P < len) P <<= 1;
    // keys of one list, or of all lists side by side where merge_lists sorts them together
    const size_t keys = (size_t) P * 12 * (P <= MERGE_JOINT_MAX ? MAX_LISTS : 1);
    return keys + (size_t) MAX_LISTS * MERGE_MAX_WANT * (4 + 2) + (size_t) HASH_SLOTS * 6 + 64;
}

// ---- the whole selection as ONE cooperative launch -------------------------------------------------------
// The launch is cooperative (all blocks resident), so the grid barriers cannot deadlock. Every block takes the same path
// through them: the decisions between them depend only on state written before the previous barrier.
namespace cg = cooperative_groups;
constexpr int SELECT_THREADS = 1024;
constexpr int SELECT_CAP = 4096;            // candidates per list that fit the buffers (and a block's shared memory)
constexpr int SAMPLE_RUN = 16;              // the sample is taken in runs of 16 instances (one 128-byte line of f)
constexpr int SAMPLE_MIN = 2048, SAMPLE_MAX = 8192;
static_assert(SELECT_THREADS == MERGE_THREADS, "the last block walks the lists");

struct SelectArgs {
    int solver_kind, n;
    const double *f, *alpha;
    const int *y;
    const unsigned char *in_ws;
    double Cp, Cn;
    SelectState *st;
    int *hist, *ticket;
    int want, id_offset;
    int sample, rank_low, rank_high;    // sample size; the pivot's rank in the sample lies in [rank_low, rank_high] if it can
    unsigned long long *cand_h;         // [lists][SELECT_CAP] keys of the candidates
    unsigned int *cand_l;
    double *sorted_f;                   // the `want` best of every list, sorted, padded with id -1: [lists][want]
    int *sorted_id;
    int *out_ids, *out_count;           // the merged selection, or nullptr: the sorted lists are the result
    const int *stop;                    // optional: when *stop is non-zero the whole launch is a no-op
    PhaseTimes *times;                  // optional
};

// Resolves one 12-bit digit of every active list from histograms of 4,096 bins each (threads 256 l .. 256 l + 255 own list
// l, 16 bins each): the digit that holds rank k_rem(l). done(l, t8, ...) is called by the one thread that finds it.
template <typename Done>
__device__ __forceinline__ void resolve_digits(int lists, unsigned active, int *hist, bool from_l2, const int (&k_rem)[MAX_LISTS],
                                               int *scan, Done done) {
    const int tid = threadIdx.x, l = tid >> 8, t8 = tid & 255, lane = tid & 31;
    const bool mine = l < lists && ((active >> l) & 1u);
    int local[16], sum = 0;
    int *h = hist + l * RADIX_BINS + t8 * 16;
    if (mine) {
#pragma unroll
        for (int b4 = 0; b4 < 16; b4 += 4) {
            const int4 v = from_l2 ? __ldcg(reinterpret_cast<const int4 *>(h + b4)) : *reinterpret_cast<const int4 *>(h + b4);
            local[b4] = v.x; local[b4 + 1] = v.y; local[b4 + 2] = v.z; local[b4 + 3] = v.w;
            sum += v.x + v.y + v.z + v.w;
        }
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
    if (lane == 31) scan[tid >> 5] = inc;              // 32 warp totals: 8 per list
    __syncthreads();
    if (mine) {
        int before = inc - sum, total = 0;
        for (int w = 0; w < 8; ++w) {
            const int v = scan[(l << 3) + w];
            if (w < (t8 >> 5)) before += v;
            total += v;
        }
        int k = 0;
#pragma unroll
        for (int x = 0; x < MAX_LISTS; ++x) if (x == l) k = k_rem[x];
        if (total < k) {
            if (t8 == 0) done(l, -1, 0, 0);
        } else if (before < k && k <= before + sum) {
            int run = before;
#pragma unroll
            for (int b = 0; b < 16; ++b) {
                if (run < k && k <= run + local[b]) done(l, t8 * 16 + b, run, local[b]);
                run += local[b];
            }
        }
    }
}

struct Pivots {                 // shared memory: candidates of list l are the eligible keys <= (h, lo)
    unsigned long long h[MAX_LISTS];
    unsigned int lo[MAX_LISTS];
    int k_rem[MAX_LISTS];
    int below[MAX_LISTS];       // sample entries below the prefix found so far
    unsigned open;              // bit l: list l is not resolved yet
};

// The pivots from the sample, the same in every block. smem: keys, list bits and the digit histograms.
__device__ void sample_pivots(const SelectArgs &a, int lists, Pivots &pv, unsigned char *smem) {
    const int tid = threadIdx.x, S = a.sample;
    unsigned long long *key = reinterpret_cast<unsigned long long *>(smem);            // [S]
    int *hist = reinterpret_cast<int *>(key + ((S + 1) & ~1));                          // [lists][RADIX_BINS], 16-byte aligned
    unsigned char *bits = reinterpret_cast<unsigned char *>(hist + lists * RADIX_BINS);  // [S]
    __shared__ int scan[32];
    auto place = [&](int i) {
        return S == a.n ? i : (int) ((long long) (i / SAMPLE_RUN) * a.n / (S / SAMPLE_RUN)) + i % SAMPLE_RUN;
    };
    for (int i = tid; i < S; i += SELECT_THREADS) {
        const int j = place(i);
        const unsigned m = lists_of(a.solver_kind, a.alpha[j], a.y[j], a.Cp, a.Cn);
        key[i] = ordered_key(a.f[j]);
        bits[i] = (unsigned char) (a.in_ws && a.in_ws[j] ? 0u : m);
    }
    if (tid < MAX_LISTS) { pv.h[tid] = 0; pv.lo[tid] = 0; pv.k_rem[tid] = a.rank_low; pv.below[tid] = 0; }
    if (tid == 0) pv.open = (1u << lists) - 1;
    for (int pass = 0; pass < RADIX_PASSES; ++pass) {
        for (int b = tid; b < lists * RADIX_BINS; b += SELECT_THREADS) hist[b] = 0;
        __syncthreads();
        const unsigned open = pv.open;
        if (!open) break;
        const int shift = 96 - RADIX_BITS * (pass + 1);
        for (int i0 = 0; i0 < S; i0 += SELECT_THREADS) {            // whole warps enter every round
            const int i = i0 + tid;
            const unsigned m = i < S ? bits[i] & open : 0u;
            const unsigned long long k0 = i < S ? key[i] : 0ull;
            const unsigned id = i < S ? (unsigned) place(i) : 0u;
#pragma unroll
            for (int l = 0; l < MAX_LISTS; ++l) {
                if (l >= lists) continue;
                const bool asc = list_ascending(a.solver_kind, l);
                const key96_t k = ((key96_t) (asc ? k0 : ~k0) << 32) | (asc ? id : ~id);
                const key96_t prefix = ((key96_t) pv.h[l] << 32) | pv.lo[l];
                const bool hit = ((m >> l) & 1u) && (pass == 0 || (k >> (shift + RADIX_BITS)) == (prefix >> (shift + RADIX_BITS)));
                const int digit = (int) (k >> shift) & (RADIX_BINS - 1);
                if (pass == 0) {
                    // (sign and exponent: few different digits, so one addition per digit and warp)
                    const unsigned peers = __match_any_sync(0xffffffffu, hit ? digit : -1);
                    if (hit && (int) (tid & 31) == __ffs(peers) - 1) atomicAdd(&hist[l * RADIX_BINS + digit], __popc(peers));
                } else if (hit) atomicAdd(&hist[l * RADIX_BINS + digit], 1);
            }
        }
        __syncthreads();
        int k_rem[MAX_LISTS];
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l) k_rem[l] = pv.k_rem[l];
        resolve_digits(lists, open, hist, false, k_rem, scan, [&](int l, int digit, int before, int inside) {
            if (digit < 0) {                                        // too few in the sample: take every eligible instance
                pv.h[l] = ~0ull; pv.lo[l] = ~0u;
                atomicAnd(&pv.open, ~(1u << l));
                return;
            }
            key96_t p = (((key96_t) pv.h[l] << 32) | pv.lo[l]) | ((key96_t) digit << shift);
            if (shift == 0 || pv.below[l] + before + inside <= a.rank_high) {
                p |= ((key96_t) 1 << shift) - 1;
                atomicAnd(&pv.open, ~(1u << l));
            }
            pv.h[l] = (unsigned long long) (p >> 32); pv.lo[l] = (unsigned) p;
            pv.k_rem[l] -= before;
            pv.below[l] += before;
        });
        __syncthreads();
    }
    __syncthreads();
}

// Exact pivots of all lists by a radix select over all instances (grid barriers inside; every block calls it).
__device__ void exact_pivots(const SelectArgs &a, int lists, Pivots &pv, cg::grid_group &grid, unsigned char *smem) {
    int *sh = reinterpret_cast<int *>(smem);
    __shared__ int scan[32];
    __shared__ bool is_last;
    volatile SelectState *st = a.st;        // written by other blocks between the barriers: always read from L2
    const int tid = threadIdx.x, gtid = blockIdx.x * SELECT_THREADS + tid, gsize = gridDim.x * SELECT_THREADS;
    for (int i = gtid; i < lists * RADIX_BINS; i += gsize) a.hist[i] = 0;
    if (gtid < lists) {
        st[gtid].prefix_hi = 0; st[gtid].prefix_lo = 0; st[gtid].k_rem = a.want; st[gtid].take_all = 0;
        st[gtid].count = 0; st[gtid].resolved = 0;
    }
    if (gtid == 0) *a.ticket = 0;
    grid.sync();
    for (int pass = 0; pass < RADIX_PASSES; ++pass) {
        const int shift = 96 - RADIX_BITS * (pass + 1);
        unsigned active = 0;
        key96_t prefix[MAX_LISTS];
        int k_rem[MAX_LISTS];
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l) {
            prefix[l] = 0; k_rem[l] = 0;
            if (l < lists && !st[l].take_all && !st[l].resolved) {
                active |= 1u << l;
                prefix[l] = ((key96_t) st[l].prefix_hi << 32) | st[l].prefix_lo;
                k_rem[l] = st[l].k_rem;
            }
        }
        if (!active) break;                      // the same for every block: the state was final before the barrier
        for (int b = tid; b < lists * RADIX_BINS; b += SELECT_THREADS) sh[b] = 0;
        __syncthreads();
        for (int j = gtid; j < a.n; j += gsize) {
            if (a.in_ws && a.in_ws[j]) continue;
            const double al = a.alpha[j], fj = a.f[j];
            const int yj = a.y[j];
#pragma unroll
            for (int l = 0; l < MAX_LISTS; ++l) {
                if (!((active >> l) & 1u)) continue;
                if (!in_list(a.solver_kind, l, al, yj, a.Cp, a.Cn)) continue;
                const key96_t k = make_key(list_ascending(a.solver_kind, l), fj, (unsigned) j);
                if (pass > 0 && (k >> (shift + RADIX_BITS)) != (prefix[l] >> (shift + RADIX_BITS))) continue;
                const int bin = l * RADIX_BINS + ((int) (k >> shift) & (RADIX_BINS - 1));
                if (pass == 0) {
                    const unsigned peers = __match_any_sync(__activemask(), bin);
                    if ((int) (tid & 31) == __ffs(peers) - 1) atomicAdd(&sh[bin], __popc(peers));
                } else {
                    atomicAdd(&sh[bin], 1);
                }
            }
        }
        __syncthreads();
        for (int b = tid; b < lists * RADIX_BINS; b += SELECT_THREADS)
            if (sh[b]) atomicAdd(&a.hist[b], sh[b]);
        __threadfence();
        __syncthreads();
        if (tid == 0) is_last = (atomicAdd(a.ticket, 1) == (int) gridDim.x - 1);
        __syncthreads();
        if (is_last) {                           // the last block to finish its sweep picks the digits
            __threadfence();
            resolve_digits(lists, active, a.hist, true, k_rem, scan, [&](int l, int digit, int before, int inside) {
                if (digit < 0) { st[l].take_all = 1; return; }       // can only happen in pass 0
                key96_t p = 0;
                int k = 0;
#pragma unroll
                for (int x = 0; x < MAX_LISTS; ++x) if (x == l) { p = prefix[x]; k = k_rem[x] - before; }
                p |= (key96_t) digit << shift;
                if (shift == 0 || (a.want - k) + inside <= SELECT_CAP) {
                    p |= ((key96_t) 1 << shift) - 1;
                    st[l].resolved = 1;
                }
                st[l].prefix_hi = (unsigned long long) (p >> 32);
                st[l].prefix_lo = (unsigned int) p;
                st[l].k_rem = k;
            });
            __syncthreads();
            for (int b = tid; b < lists * RADIX_BINS; b += SELECT_THREADS) a.hist[b] = 0;
            if (tid == 0) *a.ticket = 0;
            __threadfence();
        }
        grid.sync();
    }
    if (tid < lists) {
        pv.h[tid] = st[tid].take_all ? ~0ull : st[tid].prefix_hi;
        pv.lo[tid] = st[tid].take_all ? ~0u : st[tid].prefix_lo;
    }
    __syncthreads();
}

// Candidates of every list (eligible keys up to the pivot) into cand_*; st[l].count counts them, beyond SELECT_CAP too.
__device__ void collect_candidates(const SelectArgs &a, int lists, const Pivots &pv) {
    const int lane = threadIdx.x & 31, gtid = blockIdx.x * SELECT_THREADS + threadIdx.x, gsize = gridDim.x * SELECT_THREADS;
    for (int j0 = gtid - lane; j0 < a.n; j0 += gsize) {          // whole warps enter every round (ballots below)
        const int j = j0 + lane;
        const bool live = j < a.n;
        const int jc = live ? j : a.n - 1;
        unsigned m = lists_of(a.solver_kind, a.alpha[jc], a.y[jc], a.Cp, a.Cn);
        const unsigned long long key = ordered_key(a.f[jc]);
        if (!live || (a.in_ws && a.in_ws[jc])) m = 0;
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l) {
            if (l >= lists) continue;
            const bool asc = list_ascending(a.solver_kind, l);
            const unsigned long long h = asc ? key : ~key;
            const unsigned lo = asc ? (unsigned) j : ~(unsigned) j;
            const bool hit = ((m >> l) & 1u) && (h < pv.h[l] || (h == pv.h[l] && lo <= pv.lo[l]));
            const unsigned peers = __ballot_sync(0xffffffffu, hit);
            if (!peers) continue;
            int base = 0;                                         // one atomic per warp and list
            if (lane == __ffs(peers) - 1) base = atomicAdd(&a.st[l].count, __popc(peers));
            base = __shfl_sync(0xffffffffu, base, __ffs(peers) - 1);
            const int pos = base + __popc(peers & ((1u << lane) - 1));
            if (hit && pos < SELECT_CAP) {
                a.cand_h[(size_t) l * SELECT_CAP + pos] = h;
                a.cand_l[(size_t) l * SELECT_CAP + pos] = lo;
            }
        }
    }
}

__global__ void __launch_bounds__(SELECT_THREADS, 1) select_kernel(const SelectArgs a) {
    extern __shared__ __align__(16) unsigned char select_smem[];
    __shared__ Pivots pv;
    __shared__ bool is_last;
    cg::grid_group grid = cg::this_grid();
    const int lists = list_count(a.solver_kind);
    const int tid = threadIdx.x, lane = tid & 31;
    // written by an earlier launch only: every thread of every block reads the same value and leaves before
    // the first grid barrier
    if (a.stop && *a.stop) return;
    if (a.times && blockIdx.x == 0 && tid == 0) a.times->select_begin = device_ns();

    sample_pivots(a, lists, pv, select_smem);
    collect_candidates(a, lists, pv);
    grid.sync();
    int count[MAX_LISTS];
    bool typical = true;
#pragma unroll
    for (int l = 0; l < MAX_LISTS; ++l) {
        count[l] = l < lists ? __ldcg(&a.st[l].count) : 0;
        const bool all = l < lists && pv.h[l] == ~0ull;           // every eligible instance was taken
        if (l < lists && (count[l] > SELECT_CAP || (count[l] < a.want && !all))) typical = false;
    }
    if (!typical) {
        grid.sync();                                              // everyone has read the counts that are reset now
        exact_pivots(a, lists, pv, grid, select_smem);
        collect_candidates(a, lists, pv);
        grid.sync();
#pragma unroll
        for (int l = 0; l < MAX_LISTS; ++l) count[l] = l < lists ? __ldcg(&a.st[l].count) : 0;
    }

    // A candidate's place in its sorted list is the number of smaller keys: one warp per candidate, all candidates of
    // the list in shared memory. (12 KB per list at a thousand candidates; a bitonic sort of two such lists by one
    // block took 25 us, this takes 3.)
    unsigned long long *kh = reinterpret_cast<unsigned long long *>(select_smem);       // [SELECT_CAP]
    unsigned int *kl = reinterpret_cast<unsigned int *>(kh + SELECT_CAP);
    const int gwarp = (blockIdx.x * SELECT_THREADS + tid) >> 5, n_warps = (gridDim.x * SELECT_THREADS) >> 5;
    for (int l = 0; l < lists; ++l) {
        const int c = count[l];
        const bool asc = list_ascending(a.solver_kind, l);
        __syncthreads();
        for (int e = tid; e < c; e += SELECT_THREADS) {
            kh[e] = __ldcg(a.cand_h + (size_t) l * SELECT_CAP + e);
            kl[e] = __ldcg(a.cand_l + (size_t) l * SELECT_CAP + e);
        }
        __syncthreads();
        // (the lists start at different warps, so that few candidates occupy all of them)
        for (int e = (gwarp + l * (n_warps / lists)) % n_warps; e < c; e += n_warps) {
            const unsigned long long h = kh[e];
            const unsigned lo = kl[e];
            int smaller = 0;
            for (int x = lane; x < c; x += 32) smaller += key_less(kh[x], kl[x], h, lo) ? 1 : 0;
            smaller = __reduce_add_sync(0xffffffffu, smaller);
            if (lane == 0 && smaller < a.want) {
                a.sorted_f[(size_t) l * a.want + smaller] = key_to_double(asc ? h : ~h);
                a.sorted_id[(size_t) l * a.want + smaller] = (int) (asc ? lo : ~lo) + a.id_offset;
            }
        }
        for (int e = c + gwarp * 32 + lane; e < a.want; e += n_warps * 32) {
            a.sorted_f[(size_t) l * a.want + e] = 0.0;
            a.sorted_id[(size_t) l * a.want + e] = -1;
        }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) is_last = atomicAdd(a.ticket, 1) == (int) gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (tid < lists) a.st[tid].count = 0;                         // for the next call
    if (tid == 0) *a.ticket = 0;
    if (!a.out_ids) return;

    // the last block to finish merges the lists
    int *top_id = reinterpret_cast<int *>(select_smem);                                  // [lists][MERGE_MAX_WANT]
    short *partner = reinterpret_cast<short *>(top_id + MAX_LISTS * MERGE_MAX_WANT);
    int *hash_id = reinterpret_cast<int *>(partner + MAX_LISTS * MERGE_MAX_WANT);
    short *hash_pos = reinterpret_cast<short *>(hash_id + HASH_SLOTS);
    __shared__ int top_len[MAX_LISTS];
    __shared__ unsigned long long last_fkey[MAX_LISTS];
    for (int l = 0; l < lists; ++l)
        for (int e = tid; e < a.want; e += SELECT_THREADS) {
            top_id[l * MERGE_MAX_WANT + e] = __ldcg(a.sorted_id + (size_t) l * a.want + e);
            partner[l * MERGE_MAX_WANT + e] = -1;
        }
#pragma unroll
    for (int l = 0; l < MAX_LISTS; ++l)
        if (l < lists && tid == l) {
            const int len = count[l] < a.want ? count[l] : a.want;
            top_len[l] = len;
            last_fkey[l] = len > 0 ? ordered_key(__ldcg(a.sorted_f + (size_t) l * a.want + len - 1)) : 0ull;
        }
    __syncthreads();
    walk_lists(lists, a.want, top_id, partner, hash_id, hash_pos, top_len, last_fkey, a.out_ids, a.out_count);
}

// Sample size: all instances of small problems; else one in 128 at least, which puts the wanted 512 at about the 5th place
// of the sample and the pivot at the 15th. 8,192 at most (a block's shared memory); beyond a million instances the
// pivot is looser, not wrong.
static int select_sample(int n) {
    if (n <= SAMPLE_MIN) return n;
    int s = SAMPLE_MIN;
    while (s < n / 128 && s < SAMPLE_MAX) s *= 2;
    return s;
}
// Blocks. The sweep wants one per 2,048 instances; the rank count wants warps, about one for every 32 pairs of keys a
// small problem has to compare - up to 64 blocks, beyond which the barriers cost what the ranks save. Measured on B200,
// 512 ids (1,012 instances: of 506 eligible and up), microseconds per call with the launch, C / nu; before: every block
// at several grid barriers, one block sorting and walking the lists:
//   instances      1,012     3,000     10,000    20,242    60,000    200,000
//   before         111/133   60/135    62/96     78/110    70/125    106/170
//   now             21/27    21/34     25/36     25/35     27/37      35/45
// (all f equal, as at the start of a solve: 56 .. 192 before, 19 .. 55 now)
static int select_grid(int n) {
    const int ranks = n / 16 < 16 ? 16 : (n / 16 > 64 ? 64 : n / 16);
    const int sweep = (n + 2 * SELECT_THREADS - 1) / (2 * SELECT_THREADS);
    return sweep > ranks ? sweep : ranks;
}
static size_t select_smem_bytes(int lists, int sample) {
    const size_t pivots = (size_t) (sample + 1) * 9 + (size_t) lists * RADIX_BINS * sizeof(int);
    const size_t ranks = (size_t) SELECT_CAP * 12;
    const size_t walk = (size_t) MAX_LISTS * MERGE_MAX_WANT * (4 + 2) + (size_t) HASH_SLOTS * 6;
    const size_t most = pivots > ranks ? pivots : ranks;
    return most > walk ? most : walk;
}

}  // namespace tsvm
