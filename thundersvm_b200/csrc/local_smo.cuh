// The local solver: SMO on one working set of at most 1,024 instances, one CTA.
// Reference behaviour: c_smo_solve_kernel of the CPU backend (src/thundersvm/kernel/smo_kernel.cpp:12-125) with ties
// to the lowest slot, and nu_smo_solve_kernel of the CUDA backend (src/thundersvm/kernel/smo_kernel.cu:118-252): bound
// held in float, float arithmetic in the curvature term.
//
// What bounds it: a chain of dependent steps, about a thousand of them per call. One iteration is
//   argmin of f over I_up -> row i of the ws x ws block -> second-order argmax over I_low -> row j -> f update
// and nothing of the next iteration can start before f is updated. The two rows come from L2; the two reductions cross
// the block. So the kernel is laid out for latency: few warps with many slots each (the slots of a thread overlap, and
// what every warp has to repeat - the reductions, the step - is repeated by few warps), one barrier per reduction,
// and everything that is not on the chain is placed into the shadow of a row load.
//   * The first argmin compares the doubles themselves inside a thread and between warps; inside a warp one float
//     reduction over the doubles' high words finds the winner, and only if two lanes share the high word the low words
//     are looked at.
//   * The largest f over I_low is needed for the stopping rule only. Its high word gives a lower bound of it; the
//     exact value is reduced when the bound cannot show that the gap is still open.
//   * The second-order values b^2 / a are compared in FP32 (error below 1e-6 relative: b truncated to 24 bits, a rounded
//     once, an approximate reciprocal). If the best value of the block stands out by more than 8e-6 it is the
//     winner in FP64 too; otherwise - near-equal instances, mostly - or if an operand leaves the range in which that
//     error bound holds, the block repeats the comparison in FP64 (a few ulp), ties to the lower slot.
// Measured (RBF block, 1,024 slots): 1.00 us per iteration, 1.74 before (512 threads with two slots each, every mirror
// written in every iteration, FP64 keys and one exact division per thread in the second-order choice); where most
// values tie (a kernel close to the identity) 1.39 against 2.07; nu 1.48 against 2.58. Of the 1,900 cycles about 740 are
// the two L2 round trips (372 cycles each), 440 the first reduction, 250 the second. Inside a solve, where other kernels use
// the L2, the rows copied ahead (copy_rows_ahead) count more: 10,000 x 20 339 -> 307 us per call, next to the kernel-row
// launch of 200,000 x 2,000 817 -> 597 us.
#pragma once
#include "common.cuh"

namespace tsvm {

constexpr int NO_SLOT = 0x7fffffff;

namespace smo {
constexpr float FAR_POS = 1.7014118e38f;                            // as the high word of a double: 2^1008
constexpr double NO_MEMBER = 1e300;                                 // |value| above it: no instance in the list

__device__ __forceinline__ float high_as_float(double v) { return __int_as_float(__double2hiint(v)); }
__device__ __forceinline__ double with_high(float h, double v) { return __hiloint2double(__float_as_int(h), __double2loint(v)); }
__device__ __forceinline__ float warp_min_f32(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max_f32(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// 1 / a to a few ulp: two Newton steps on the hardware's approximation (which is kept for zero and infinity)
__device__ __forceinline__ double reciprocal(double a) {
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(a));
    double r = fma(r0, fma(-a, r0, 1.0), r0);
    r = fma(r, fma(-a, r, 1.0), r);
    return a != 0.0 && fabs(a) < 1e300 ? r : r0;
}

// Row ring: rows of kww that the next iterations are likely to need, copied to shared memory by a warp of its own.
constexpr int RING = 32;                // one ring slot per lane of the copying warp
constexpr int RING_SPARE = 10;          // slots kept free for the next copies
constexpr int NOT_THERE = -1, ON_THE_WAY = -2;

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned) __cvta_generic_to_shared(p); }
__device__ __forceinline__ int load_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void store_release(int *p, int v) {
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}
__device__ __forceinline__ bool copy_done(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
template <int T>
__device__ __forceinline__ void solver_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory"); }

struct First { double f; int slot; float low; };        // a warp's smallest f over I_up, its slot; high word of max f over I_low
struct Second { float best, next; int slot, pad; };     // a warp's largest and second-largest estimate of b^2 / a

// The copying warp. Which rows the next iterations need can be guessed: the winner of an argmin is usually among the best
// few of the argmin before. Every warp of the solver leaves its best two slots of both argmins in `cand` (n_cand ids);
// whichever of them has no row in the ring is copied there, and a row that has not been wanted for longest makes room.
//   where[t]: ring slot of row t, NOT_THERE or ON_THE_WAY. It is set only when the copy has arrived, so a solver thread
//   either finds the row or reads kww; both hold the same values. The copying warp's wait on the mbarrier makes the row
//   visible to itself; its release of `where` and the solver threads' acquire pass that on.
//   A row is taken out of `where` first, and the fence before `window` is read has that seen by the whole block; its slot is
//   overwritten three windows later (a window: from one barrier of the solver to the next). A row that a solver thread finds
//   in a window is read in that window and the next; the barrier orders those reads before thread 0's release of a later
//   `window`, which the copying warp acquires before it copies.
//   Measured: the two acquires and the two releases cost 0.5 - 1 % of a solve (10,000 x 20: 33.9 -> 34.3 ms). Letting thread 0
//   read a count of removals and hand it back with `window` cost 2 - 3 % more.
__device__ void copy_rows_ahead(const float *__restrict__ kww, int ws, float *ring, int *where, const int *cand, int n_cand,
                                const int *window, const int *done, unsigned long long *bars, int *stamp, int *stage) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu, bar = smem_addr(bars + lane), row_bytes = (unsigned) ws * 4;
    enum { FREE, COMING, READY };
    int state = FREE, row = 0, freed = -4, used = 0, seen = -1;
    unsigned parity = 0;
    auto arrived = [&](int now) {
        if (state == COMING && copy_done(bar, parity)) {
            parity ^= 1;
            state = READY;
            used = now;
            store_release(where + row, lane);
        }
    };
    // (bounded: a solver that runs longer than this goes on without new rows)
    for (int polls = 0; polls < (1 << 26); ++polls) {
        const int now = load_acquire(window);
        if (load_acquire(done)) break;
        arrived(now);
        if (__all_sync(full, now == seen)) { __nanosleep(32); continue; }
        seen = now;
        // candidates without a row, each once
        const int x = lane < n_cand ? *(volatile const int *) (cand + lane) : -1;
        const bool valid = (unsigned) x < (unsigned) ws;
        const int at = valid ? *(volatile int *) (where + x) : (int) ON_THE_WAY;
        const unsigned same = __match_any_sync(full, valid ? x : -1 - lane);
        const bool need = valid && at == NOT_THERE && lane == __ffs(same) - 1;
        if (valid && at >= 0) stamp[at] = now;
        const unsigned needs = __ballot_sync(full, need);
        if (need) stage[__popc(needs & ((1u << lane) - 1))] = x;
        __syncwarp();
        if (state == READY && stamp[lane] == now) used = now;
        const bool open = state == FREE && now - freed >= 3;
        const unsigned opens = __ballot_sync(full, open);
        const int k = __popc(opens & ((1u << lane) - 1));
        if (open && k < __popc(needs)) {
            row = stage[k];
            *(volatile int *) (where + row) = ON_THE_WAY;
            state = COMING;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(row_bytes) : "memory");
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_addr(ring + (size_t) lane * ws)), "l"(kww + (size_t) row * ws), "r"(row_bytes), "r"(bar) : "memory");
        }
        // make room: the row that has not been wanted for longest
        const int spare = __popc(__ballot_sync(full, state == FREE));
        const int oldest = __reduce_min_sync(full, state == READY ? used : 0x7fffffff);
        const unsigned olds = __ballot_sync(full, state == READY && used == oldest);
        if (spare < RING_SPARE && state == READY && used == oldest && oldest < now &&
            __popc(olds & ((1u << lane) - 1)) < RING_SPARE - spare) {
            store_release(where + row, NOT_THERE);
            __threadfence_block();
            state = FREE;
            freed = load_acquire(window);
        }
        __syncwarp();
    }
    for (int polls = 0; polls < (1 << 24) && __any_sync(full, state == COMING); ++polls) arrived(0);
}
}  // namespace smo

// Slot t of the working set belongs to thread t % T. S slots per thread; 32 more threads copy rows ahead.
template <bool NU, int S, int T>
__global__ void __launch_bounds__(T + 32, 1)
local_smo_kernel(int ws, const float *__restrict__ kww, const float *__restrict__ diag_ws,
                 const int *__restrict__ y_ws, const double *__restrict__ f_ws, double *__restrict__ alpha_ws,
                 double *__restrict__ alpha_diff, double Cp_in, double Cn_in, double eps, int max_iter,
                 double *__restrict__ diff, const int *__restrict__ ids, double *__restrict__ alpha_global,
                 const int *__restrict__ stop, int use_ring, PhaseTimes *times) {
    using namespace smo;
    constexpr int W = T / 32, CLS = NU ? 2 : 1;             // nu: the lists of I_up and I_low are split by class
    constexpr bool AHEAD = !NU;                             // (nu reads two rows i and guesses j badly: 5 % slower with the ring)
    if (stop && *stop) {            // queued past the end of a solve: no step, so the f update that follows adds zero
        for (int t = threadIdx.x; t < ws; t += T + 32) alpha_diff[t] = 0;
        return;
    }
    if (times && threadIdx.x == 0) times->local_begin = device_ns();
    __shared__ double f_sm[S * T], a_sm[S * T];
    __shared__ float kd_sm[S * T];
    __shared__ int y_sm[S * T];
    __shared__ First e1[CLS][W];
    __shared__ Second e2[W];
    __shared__ unsigned long long exact_key[CLS][W];
    __shared__ int exact_slot[CLS][W];
    __shared__ double exact_low[CLS][W];
    // row ring (use_ring): ring [RING][ws] floats in dynamic shared memory
    extern __shared__ __align__(128) float ring[];
    constexpr int N_CAND = 2 * (CLS + 1) * W;
    __shared__ int where[S * T], cand[N_CAND], ring_stamp[RING], ring_stage[32], window, done;
    __shared__ __align__(8) unsigned long long ring_bar[RING];
    static_assert(N_CAND <= 32, "one candidate per lane of the copying warp");
    const double Cp = NU ? (double) (float) Cp_in : Cp_in;
    const double Cn = NU ? Cp : Cn_in;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid >= T) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(ring_bar + lane)) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        ring_stamp[lane] = -1;
        if (lane < N_CAND) cand[lane] = -1;
        if (lane == 0) { window = 0; done = 0; }
        for (int t = lane; t < S * T; t += 32) where[t] = NOT_THERE;
        __syncthreads();
        if (AHEAD && use_ring) copy_rows_ahead(kww, ws, ring, where, cand, N_CAND, &window, &done, ring_bar, ring_stamp, ring_stage);
        return;
    }

    double f[S];
    float kd[S], pen_up[S], pen_low[S];     // +-FAR_POS: what clamps a non-member's f out of the list
    bool pos[S];                            // nu: class of the slot
    int off[S];                             // column of the slot in a row of kww (any valid one where there is no slot)
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int t = tid + s * T;
        double a = 0;
        int y = 0;                          // y = 0: member of no set
        f[s] = 0; kd[s] = 0;
        if (t < ws) { f[s] = f_ws[t]; a = alpha_ws[t]; y = y_ws[t]; kd[s] = diag_ws[t]; }
        f_sm[t] = f[s]; a_sm[t] = a; y_sm[t] = y; kd_sm[t] = kd[s];
        pen_up[s] = in_I_up(a, y, Cp, Cn) ? -FAR_POS : FAR_POS;
        pen_low[s] = in_I_low(a, y, Cp, Cn) ? FAR_POS : -FAR_POS;
        pos[s] = y > 0;
        off[s] = t < ws ? t : 0;
    }
    __syncthreads();
    auto read_row = [&](int r, int at, float (&k)[S]) {
        if (at >= 0) {
#pragma unroll
            for (int s = 0; s < S; ++s) k[s] = ring[at * ws + off[s]];
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) k[s] = __ldg(kww + r * ws + off[s]);
        }
    };

    double local_eps = 0;
    int it = 0;
    // the last step, written to a_sm once every thread has read what it needs for that step
    int step_i = 0, step_j = 0;
    double step_ai = a_sm[0], step_aj = step_ai;
    for (;;) {
        float first_h[CLS];                 // the lane's best, without the warp's winner
        int first_slot[CLS];
        // ---- smallest f over I_up (with its slot), high word of the largest f over I_low ---------------------
        float low_h[S];                     // high word of f, clamped to -FAR_POS outside I_low
#pragma unroll
        for (int s = 0; s < S; ++s) low_h[s] = fminf(high_as_float(f[s]), pen_low[s]);
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            double v[S];
            int slot[S];
            float lo = -FAR_POS;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float h = fmaxf(high_as_float(f[s]), pen_up[s]);
                const bool mine = !NU || pos[s] == (c == 0);
                v[s] = with_high(mine ? h : FAR_POS, f[s]);
                slot[s] = tid + s * T;
                lo = fmaxf(lo, mine ? low_h[s] : -FAR_POS);
            }
            // The warp's reduction runs over the high words and needs only their minimum; the exact minimum and its slot
            // are found next to it. Neighbouring slots first: the left operand always holds the lower slots and wins ties.
            float h = high_as_float(v[0]);
#pragma unroll
            for (int s = 1; s < S; ++s) h = fminf(h, high_as_float(v[s]));
            const float h_min = warp_min_f32(h), lo_max = warp_max_f32(lo);
#pragma unroll
            for (int d = 1; d < S; d <<= 1)
#pragma unroll
                for (int s = 0; s + d < S; s += 2 * d)
                    if (v[s + d] < v[s]) { v[s] = v[s + d]; slot[s] = slot[s + d]; }
            bool winner = h == h_min;
            First e;
            e.f = v[0]; e.slot = slot[0]; e.low = lo_max;
            if (winner) { e1[c][warp] = e; if (AHEAD) cand[c * W + warp] = slot[0]; }
            const unsigned at_min = __ballot_sync(0xffffffffu, winner);
            if (at_min & (at_min - 1)) {            // several lanes share the high word: the lane with the exact minimum writes again
                unsigned long long key = ordered_key(v[0]);
                int sl = slot[0];
                warp_argmin_u64(key, sl);
                winner = slot[0] == sl;
                __syncwarp();
                if (winner) { e1[c][warp] = e; if (AHEAD) cand[c * W + warp] = slot[0]; }
            }
            first_h[c] = winner ? FAR_POS : h;
            first_slot[c] = slot[0];
        }
        solver_barrier<T>();
        if (AHEAD && tid == 0) store_release(&window, 2 * it + 1);
        double up[CLS];
        int iu[CLS];
        float lowf[CLS];
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            double v[W];
            int slot[W];
            float lo[W];
#pragma unroll
            for (int w = 0; w < W; ++w) { const First e = e1[c][w]; v[w] = e.f; slot[w] = e.slot; lo[w] = e.low; }
#pragma unroll
            for (int d = 1; d < W; d <<= 1)
#pragma unroll
                for (int w = 0; w + d < W; w += 2 * d) {
                    lo[w] = fmaxf(lo[w], lo[w + d]);
                    if (v[w + d] < v[w] || (v[w + d] == v[w] && slot[w + d] < slot[w])) { v[w] = v[w + d]; slot[w] = slot[w + d]; }
                }
            up[c] = v[0]; iu[c] = (unsigned) slot[0] < (unsigned) ws ? slot[0] : 0; lowf[c] = lo[0];
        }
        float kI[CLS][S];
        int at_i[CLS];
#pragma unroll
        for (int c = 0; c < CLS; ++c) { at_i[c] = AHEAD ? load_acquire(where + iu[c]) : (int) NOT_THERE; read_row(iu[c], at_i[c], kI[c]); }
        // second-best lanes of the first argmin: rows to copy ahead
#pragma unroll
        for (int c = 0; c < CLS; ++c)
            if (AHEAD && first_h[c] == warp_min_f32(first_h[c])) cand[(CLS + 1 + c) * W + warp] = first_slot[c];
        // mirrors of the state after the last step (its readers have passed the barrier above)
#pragma unroll
        for (int s = 0; s < S; ++s) f_sm[tid + s * T] = f[s];
        if (tid == 0) { a_sm[step_i] = step_ai; a_sm[step_j] = step_aj; }

        // ---- stopping rule ---------------------------------------------------------------------------------
        bool open = it > 0 && it <= max_iter;
        {
            double gap = 0;
#pragma unroll
            for (int c = 0; c < CLS; ++c) {
                // the smallest double with this high word
                const int h = __float_as_int(lowf[c]);
                const double g = __hiloint2double(h, h < 0 ? -1 : 0) - up[c];
                gap = c == 0 ? g : fmax(gap, g);
            }
            open = open && gap >= local_eps;
        }
        if (!open) {
            // the exact gap: at the first iteration, near the end, and at the end
#pragma unroll
            for (int c = 0; c < CLS; ++c) {
                double m = -INFINITY;
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (pen_low[s] > 0 && (!NU || pos[s] == (c == 0))) m = fmax(m, f[s]);
                const double wm = key_to_double(~warp_min_u64(~ordered_key(m)));
                if (lane == 0) exact_low[c][warp] = wm;
            }
            solver_barrier<T>();
            double local_diff = 0;
#pragma unroll
            for (int c = 0; c < CLS; ++c) {
                double m = exact_low[c][0];
                for (int w = 1; w < W; ++w) m = fmax(m, exact_low[c][w]);
                const double d = m - (up[c] > NO_MEMBER ? INFINITY : up[c]);
                local_diff = c == 0 ? d : fmax(local_diff, d);
            }
            if (it == 0) {
                local_eps = NU ? fmax(eps, 0.1 * local_diff) : fmax(eps, (double) 0.1f * local_diff);
                if (tid == 0) diff[0] = local_diff;
            }
            if (it > max_iter || local_diff < local_eps) break;
        }

        // ---- second-order choice of j ------------------------------------------------------------------------
        float q[S], q2[S], q0[S];
        int qs[S];
        float kd_i[CLS];
#pragma unroll
        for (int c = 0; c < CLS; ++c) kd_i[c] = kd_sm[iu[c]];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const bool second = NU && !pos[s];
            const float k = second ? kI[CLS - 1][s] : kI[0][s];
            const double b = with_high(low_h[s], f[s]) - (second ? up[CLS - 1] : up[0]);    // far below zero outside I_low
            // b in FP32, truncated, straight from the double's bits; [2^-50, 2^50) keeps its square in range
            const int bh = __double2hiint(b);
            const float b32 = __int_as_float(__funnelshift_l((unsigned) __double2loint(b), (unsigned) (bh - 0x38000000), 3));
            const bool b_ok = (unsigned) (bh - 0x3cd00000) < 0x06400000u;
            const float a32 = fmaf(-2.0f, k, (second ? kd_i[CLS - 1] : kd_i[0]) + kd[s]);
            const bool a_ok = a32 > 1e-30f && a32 < 1e30f;
            float r;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a32));
            q[s] = b_ok && a_ok ? b32 * b32 * r : (b > 0 ? INFINITY : 0.0f);
            q0[s] = q[s];
            q2[s] = 0.0f;
            qs[s] = tid + s * T;
        }
#pragma unroll
        for (int d = 1; d < S; d <<= 1)
#pragma unroll
            for (int s = 0; s + d < S; s += 2 * d) {
                q2[s] = fmaxf(fminf(q[s], q[s + d]), fmaxf(q2[s], q2[s + d]));
                if (q[s + d] > q[s]) { q[s] = q[s + d]; qs[s] = qs[s + d]; }
            }
        {
            const float best = warp_max_f32(q[0]);
            const unsigned at_best = __ballot_sync(0xffffffffu, q[0] == best);
            const float mine = q[0] == best ? q2[0] : q[0];
            const float next = warp_max_f32(mine);
            if (AHEAD && mine == next && q[0] != best) cand[(2 * CLS + 1) * W + warp] = qs[0];
            if (lane == (int) __ffs(at_best) - 1) {
                Second e;
                e.best = best; e.next = (at_best & (at_best - 1)) ? best : next; e.slot = qs[0]; e.pad = 0;
                e2[warp] = e;
                if (AHEAD) cand[CLS * W + warp] = qs[0];
            }
        }
        solver_barrier<T>();
        if (AHEAD && tid == 0) store_release(&window, 2 * it + 2);
        int j;
        {
            float best[W], next[W];
            int slot[W];
#pragma unroll
            for (int w = 0; w < W; ++w) { const Second e = e2[w]; best[w] = e.best; next[w] = e.next; slot[w] = e.slot; }
#pragma unroll
            for (int d = 1; d < W; d <<= 1)
#pragma unroll
                for (int w = 0; w + d < W; w += 2 * d) {
                    next[w] = fmaxf(fminf(best[w], best[w + d]), fmaxf(next[w], next[w + d]));
                    if (best[w + d] > best[w]) { best[w] = best[w + d]; slot[w] = slot[w + d]; }
                }
            j = slot[0];
            if (!(best[0] > 0.0f && best[0] < INFINITY && next[0] < best[0] * (1.0f - 8e-6f))) {
                // too close to call in FP32, or out of its range: the same values in FP64, ties to the lower slot
                const float thr = best[0] < INFINITY ? best[0] * (1.0f - 8e-6f) : 0.0f;
                double most[CLS];
                int sl[CLS];
#pragma unroll
                for (int c = 0; c < CLS; ++c) { most[c] = -INFINITY; sl[c] = NO_SLOT; }
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const bool second = NU && !pos[s];
                    const double b = -(second ? up[CLS - 1] : up[0]) + f[s];
                    const float k = second ? kI[CLS - 1][s] : kI[0][s], kdi = second ? kd_i[CLS - 1] : kd_i[0];
                    const double a = NU ? (double) (kdi + kd[s] - 2 * k) : (double) (kdi + kd[s]) - 2.0 * (double) k;
                    const double e = b * b * reciprocal(a);
                    const bool asked = q0[s] > 0.0f && q0[s] >= thr;
#pragma unroll
                    for (int c = 0; c < CLS; ++c)
                        if (asked && second == (c > 0) && e > most[c]) { most[c] = e; sl[c] = tid + s * T; }
                }
                unsigned long long key[CLS];
#pragma unroll
                for (int c = 0; c < CLS; ++c) key[c] = ordered_key(-most[c]);
#pragma unroll
                for (int c = 0; c < CLS; ++c) {
                    warp_argmin_u64(key[c], sl[c]);
                    if (lane == 0) { exact_key[c][warp] = key[c]; exact_slot[c][warp] = sl[c]; }
                }
                solver_barrier<T>();
#pragma unroll
                for (int c = 0; c < CLS; ++c) {
                    key[c] = lane < W ? exact_key[c][lane] : ~0ull;
                    sl[c] = lane < W ? exact_slot[c][lane] : NO_SLOT;
                    warp_argmin_u64(key[c], sl[c]);
                }
                j = sl[0];
                // the positive-class pair wins only if its value is strictly smaller (smo_kernel.cu:220-233)
                if (NU && !(key_to_double(key[0]) < key_to_double(key[CLS - 1]))) j = sl[CLS - 1];
                if (j == NO_SLOT) j = 0;
            }
        }
        // ---- step, repeated by every thread in the shadow of row j -------------------------------------------
        float kJ[S];
        read_row(j, AHEAD ? load_acquire(where + j) : (int) NOT_THERE, kJ);
        const int yj = y_sm[j];
        const bool second = NU && yj < 0;
        const int i = second ? iu[CLS - 1] : iu[0];
        const int yi = y_sm[i];
        const double u = second ? up[CLS - 1] : up[0];
        const double ai = a_sm[i], aj = a_sm[j], fj = f_sm[j];
        const int at = second ? at_i[CLS - 1] : at_i[0];
        const float kij = at >= 0 ? ring[at * ws + j] : __ldg(kww + i * ws + j);      // row i has just been read: from L1
        const double room_i = yi > 0 ? Cp - ai : ai;
        const double curv = NU ? (double) (kd_sm[i] + kd_sm[j] - 2 * kij)
                               : (double) (kd_sm[i] + kd_sm[j]) - 2.0 * (double) kij;
        const double room_j = fmin(yj > 0 ? aj : Cn - aj, (-u + fj) / curv);
        const double l = fmin(room_i, room_j);
        step_i = i; step_j = j;
        step_ai = ai + l * yi; step_aj = aj - l * yj;
        const float up_i = in_I_up(step_ai, yi, Cp, Cn) ? -FAR_POS : FAR_POS, up_j = in_I_up(step_aj, yj, Cp, Cn) ? -FAR_POS : FAR_POS;
        const float lo_i = in_I_low(step_ai, yi, Cp, Cn) ? FAR_POS : -FAR_POS, lo_j = in_I_low(step_aj, yj, Cp, Cn) ? FAR_POS : -FAR_POS;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int t = tid + s * T;
            if (t == i) { pen_up[s] = up_i; pen_low[s] = lo_i; }
            if (t == j) { pen_up[s] = up_j; pen_low[s] = lo_j; }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const float k = second ? kI[CLS - 1][s] : kI[0][s];
            const double d = NU ? (double) (kJ[s] - k) : (double) kJ[s] - (double) k;
            f[s] = fma(-l, d, f[s]);
        }
        ++it;
    }
    if (tid == 0) store_release(&done, 1);
    solver_barrier<T>();            // (the last step's alphas are in a_sm)
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int t = tid + s * T;
        if (t < ws) {
            const double a = a_sm[t], a_old = alpha_ws[t];
            alpha_ws[t] = a;
            alpha_diff[t] = -(a - a_old) * y_sm[t];
            if (alpha_global && ids[t] >= 0) alpha_global[ids[t]] = a;
        }
    }
    if (tid == 0) {
        diff[1] = it;
        if (times) times->local_end = device_ns();
    }
}

}  // namespace tsvm
