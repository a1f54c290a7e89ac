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
//     exact value is reduced when the bound cannot show that the gap is still open. The rule is applied after the second
//     argmin, next to the loads for the step: nothing has been changed by then.
//   * The second-order values b^2 / a are compared in FP32 (error below 1e-6 relative: b truncated to 24 bits, a rounded
//     once, an approximate reciprocal). If the best value of the block stands out by more than 8e-6 it is the
//     winner in FP64 too; otherwise - near-equal instances, mostly - or if an operand leaves the range in which that
//     error bound holds, the block repeats the comparison in FP64 (a few ulp), ties to the lower slot.
//   * No conversion instructions on the chain (16 of them took 160 cycles): f is held times 2^-896, which makes a float's
//     bits a double's and a double's a float's by shifts. A value of f below 2^-126 loses digits that way, sums of kernel
//     values do not get there.
//   * The step is divided by a reciprocal after one Newton-Raphson iteration, the quotient corrected by its remainder: the method
//     of P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor" (IBM Journal of Research and
//     Development 34, 1990), which rests on the fused multiply-add. Within an ulp of the division: the hardware's approximation of
//     the reciprocal has some 20 bits, the iteration squares its error, and the correction squares that (below 2^-70, beside the last
//     rounding).
//   * Two more warps read the rows that the next iterations will want into the L1 cache (read_rows_ahead). In most calls every
//     row is wanted about once, so a cache alone finds a tenth of them; the best six of an argmin's list hold the next
//     iteration's winner nine times in ten.
// Measured per iteration at 1,024 slots inside a solve, before (conversions, an exact division, 32 rows copied to shared
// memory by one more warp and looked up there) and now: 10,000 x 20 1.05 -> 0.82 us, 12,003 x 784 1.00 -> 0.81, text
// 1.00 -> 0.80, one-hot records, where many values tie, 1.10 -> 0.88, 200,000 x 2,000 next to the kernel-row launch
// 1.44 -> 1.20, nu (without the reading warps) 1.38 -> 1.15. With every row found in L1 an iteration takes 0.67 us: 486
// instructions per warp (604 before) at 2.7 cycles, dependent ones mostly. Two floats per instruction in the second-order
// values (16 instructions fewer) changed nothing; masks instead of compares where a slot joins or leaves a list cost 5 %.
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

// 1 / a to a few ulp: two Newton-Raphson iterations r (2 - a r) on the hardware's approximation (which is kept for zero and
// infinity), each with its residual by a fused multiply-add
__device__ __forceinline__ double reciprocal(double a) {
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(a));
    double r = fma(r0, fma(-a, r0, 1.0), r0);
    r = fma(r, fma(-a, r, 1.0), r);
    return a != 0.0 && fabs(a) < 1e300 ? r : r0;
}

// Reading ahead: how many slots of an argmin are looked after, how many rows are read at a time at most, and for how many
// iterations a row that was read is taken to be there (the cache does not keep it for long): KEEP 0 / 1 / 3 make 0.821 / 0.806 /
// 0.825 us (12,003 x 784), 4 or 8 slots 0.815 or 0.819.
constexpr int KEEP = 1, WANTED = 6, MOST = 8;
template <int T>
__device__ __forceinline__ void solver_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory"); }

// What a warp leaves for the others
struct __align__(16) First { double f; int slot, pad; };            // its smallest f over I_up and that slot
struct __align__(16) Second { float best; int slot; float low[2]; };    // its largest estimate of b^2 / a; max f over I_low (high word, per class)
constexpr int SLOT_MASK = 0x7ff, TIED = 0x800;                      // TIED: another value of the warp is too close

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max_abs3(float a, float b, float c) {        // NaN if one of them is
    float r;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
template <int S>
__device__ __forceinline__ float max_of(const float (&v)[S]) {
    if constexpr (S == 8) return max3(max3(v[0], v[1], v[2]), max3(v[3], v[4], v[5]), fmaxf(v[6], v[7]));
    if constexpr (S == 4) return max3(v[0], v[1], fmaxf(v[2], v[3]));
    if constexpr (S == 2) return fmaxf(v[0], v[1]);
    return v[0];
}
template <int S>
__device__ __forceinline__ float min_of(const float (&v)[S]) {
    if constexpr (S == 8) return min3(min3(v[0], v[1], v[2]), min3(v[3], v[4], v[5]), fminf(v[6], v[7]));
    if constexpr (S == 4) return min3(v[0], v[1], fminf(v[2], v[3]));
    if constexpr (S == 2) return fminf(v[0], v[1]);
    return v[0];
}
template <int S>
__device__ __forceinline__ float max_abs_of(const float (&v)[S]) {
    if constexpr (S == 8) return max_abs3(max_abs3(v[0], v[1], v[2]), max_abs3(v[3], v[4], v[5]), max_abs3(v[6], v[7], v[7]));
    if constexpr (S == 4) return max_abs3(v[0], v[1], max_abs3(v[2], v[3], v[3]));
    return max_abs3(v[0], v[S - 1], v[S - 1]);
}
__device__ __forceinline__ float mul_ftz(float a, float b) {
    float r;
    asm("mul.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// k * 2^-896, exact for every finite float (denormals and zeros too): the float's bits, moved to where a double has them
constexpr double DOWN = 0x1p-896, BACK = 0x1p896;
__device__ __forceinline__ double widened(float k) {
    const int u = __float_as_int(k);
    return __hiloint2double((u >> 3) & 0x8fffffff, u << 29);
}

// The reading warps, one for each argmin. Every thread of the solver leaves the best of its slots (best: value, slot); the rows
// of those that are closest to the best of all are read, unless that was just done.
// A row is read by one word of each of its 32-byte sectors, by loads whose results are looked at when the next rows are read.
// (Asynchronous copies, which need no registers, take 160 cycles a row to issue against 20: a pass over six rows then lasts
// 1.7 iterations, and 60 - 75 % of the rows are found instead of 83 - 96 %; prefetch.global.L1 has no effect.)
// Nothing but time depends on what these warps see: `best`, `window` and `last` are read while they are written. A slot in
// `best` is one at any time, and no row past ws is read.
template <int S, int T, bool LARGEST>
__device__ void read_rows_ahead(const float *__restrict__ kww, int ws, const float2 *best, const int *window, const int *done,
                                int *last, int *stage) {
    constexpr int E = T / 32, G = S * T > 256 ? S * T / 256 : 1;
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    int seen = 0;
    float width = LARGEST ? 0.5f : 1e-3f;
    int used = 0, word[MOST][G] = {};
    // (bounded: a solver that runs longer than this goes on without)
    for (int polls = 0; polls < (1 << 26); ++polls) {
        const int now = *(volatile const int *) window;
        if (__any_sync(full, *(volatile const int *) done)) break;
        if (__all_sync(full, now == seen)) continue;
        seen = now;
        float v[E];
        int x[E], before[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float2 b = best[e * 32 + lane];
            // the first argmin's values are the high words of doubles
            v[e] = LARGEST ? b.x : (float) (__hiloint2double(__float_as_int(b.x), 0) * BACK);
            x[e] = __float_as_int(b.y);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) before[e] = last[x[e]];
        float m = v[0];
#pragma unroll
        for (int e = 1; e < E; ++e) m = LARGEST ? fmaxf(m, v[e]) : fminf(m, v[e]);
        m = LARGEST ? warp_max_f32(m) : warp_min_f32(m);
        // the narrowest of five widths around the last one that has WANTED slots in it
        const float unit = (LARGEST ? m : 1.0f) * width * 0.25f;
        int level = 4;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            int count = 0;
#pragma unroll
            for (int e = 0; e < E; ++e) count += fabsf(v[e] - m) <= unit * (float) (1 << k);
            if (__reduce_add_sync(full, count) >= WANTED) level = k;
        }
        const float limit = unit * (float) (1 << level);
        int n = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool need = fabsf(v[e] - m) <= limit && now - before[e] > KEEP && x[e] < ws;
            const unsigned needs = __ballot_sync(full, need);
            const int k = n + __popc(needs & ((1u << lane) - 1));
            if (need && k < MOST) { stage[k] = x[e]; last[x[e]] = now; }
            n += __popc(needs);
        }
        __syncwarp();
        // one word of every sector of 32 bytes; the words of the pass before have arrived (they are used for that alone)
#pragma unroll
        for (int k = 0; k < MOST; ++k) {
#pragma unroll
            for (int g = 0; g < G; ++g) used |= word[k][g];
            if (k < n) {
                const int *row = (const int *) kww + stage[k] * ws + lane * 8;
#pragma unroll
                for (int g = 0; g < G; ++g)
                    if (g * 256 + lane * 8 < ws) word[k][g] = __ldg(row + g * 256);
            }
        }
        width = LARGEST ? fminf(limit / m, 1.0f) : limit;
    }
    if (used == -1) last[0] = 0;            // (the loads have a use)
}
}  // namespace smo

// Slot t of the working set belongs to thread t % 32 of warp t / (32 S): a warp holds a run of 32 S slots, so that of equal
// values the lower slot is in the lower warp. S slots per thread; in the C form two more warps read rows ahead.
// f is held as f * 2^-896: a float's bits are then a double's without a conversion (widened), and a double's are a float's.
template <bool NU, int S, int T>
__global__ void __launch_bounds__(T + (NU ? 0 : 64), 1)
local_smo_kernel(int ws, const float *__restrict__ kww, const float *__restrict__ diag_ws,
                 const int *__restrict__ y_ws, const double *__restrict__ f_ws, double *__restrict__ alpha_ws,
                 double *__restrict__ alpha_diff, double Cp_in, double Cn_in, double eps, int max_iter,
                 double *__restrict__ diff, const int *__restrict__ ids, double *__restrict__ alpha_global,
                 const int *__restrict__ stop, int ahead, PhaseTimes *times) {
    using namespace smo;
    constexpr int W = T / 32, CLS = NU ? 2 : 1;             // nu: the lists of I_up and I_low are split by class
    constexpr int RUN = 32 * S;                             // slots of a warp
    if (stop && *stop) {            // queued past the end of a solve: no step, so the f update that follows adds zero
        for (int t = threadIdx.x; t < ws; t += blockDim.x) alpha_diff[t] = 0;
        return;
    }
    if (times && threadIdx.x == 0) times->local_begin = device_ns();
    __shared__ __align__(16) double f_sm[S * T];
    __shared__ double a_sm[S * T];
    __shared__ float2 ky_sm[S * T];                         // diagonal, label
    __shared__ First e1[CLS][W];
    __shared__ Second e2[W];
    __shared__ unsigned long long exact_key[CLS][W];
    __shared__ int exact_slot[CLS][W];
    __shared__ double exact_low[CLS][W];
    // what the reading warps look at: every thread's best value of the two argmins with its slot; when it changed
    constexpr bool AHEAD = !NU;                             // (nu: 1.14 us without, 1.24 with three such warps)
    __shared__ float2 best[2][T];
    __shared__ int last[S * T], window[2], done;
    __shared__ int stage[2][MOST];
    static_assert(S * T <= SLOT_MASK, "a slot fits its field");
    const double Cp = NU ? (double) (float) Cp_in : Cp_in;
    const double Cn = NU ? Cp : Cn_in;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (AHEAD && tid >= T) {
        for (int t = tid - T; t < S * T; t += 64) last[t] = -KEEP - 1;
        for (int t = tid - T; t < 2 * T; t += 64) best[0][t] = make_float2(0.0f, 0.0f);
        if (tid == T) { window[0] = window[1] = 0; done = 0; }
        __syncthreads();
        if (ahead) {
            if (warp == W) read_rows_ahead<S, T, false>(kww, ws, best[0], &window[0], &done, last, stage[0]);
            else read_rows_ahead<S, T, true>(kww, ws, best[1], &window[1], &done, last, stage[1]);
        }
        return;
    }

    // the thread's slots: runs of V, 32 V apart
    constexpr int V = NU && S >= 4 ? 4 : 1;
    const int t0 = warp * RUN + lane * V;
    auto nth = [](int s) { return s / V * (32 * V) + s % V; };
    double f[S];
    float kd[S], pen_up[CLS][S], pen_low[S];    // +-FAR_POS: what clamps a non-member's f out of the list
    bool pos[S];                            // nu: class of the slot
    float kd_most = 0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int t = t0 + nth(s);
        double a = 0;
        int y = 0;                          // y = 0: member of no set
        f[s] = 0; kd[s] = 0;
        if (t < ws) { f[s] = f_ws[t] * DOWN; a = alpha_ws[t]; y = y_ws[t]; kd[s] = diag_ws[t]; }
        f_sm[t] = f[s]; a_sm[t] = a; ky_sm[t] = make_float2(kd[s], __int_as_float(y));
        const float up_s = in_I_up(a, y, Cp, Cn) ? -FAR_POS : FAR_POS;
#pragma unroll
        for (int c = 0; c < CLS; ++c) pen_up[c][s] = !NU || (y > 0) == (c == 0) ? up_s : FAR_POS;
        pen_low[s] = in_I_low(a, y, Cp, Cn) ? FAR_POS : -FAR_POS;
        pos[s] = y > 0;
        kd_most = max_abs3(kd_most, kd[s], kd[s]);
    }
    __syncthreads();
    const bool whole = ws == S * T && (V == 1 || ((unsigned long long) kww & 15) == 0);
    auto read_row = [&](int r, float (&k)[S]) {
        const float *p = kww + r * ws + t0;
        if (whole) {
            if constexpr (V == 4) {
#pragma unroll
                for (int s = 0; s < S; s += 4) {
                    const float4 x = __ldg((const float4 *) (p + nth(s)));
                    k[s] = x.x; k[s + 1] = x.y; k[s + 2] = x.z; k[s + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int s = 0; s < S; ++s) k[s] = __ldg(p + nth(s));
            }
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) k[s] = t0 + nth(s) < ws ? __ldg(p + nth(s)) : 0.0f;
        }
    };
    const bool mild = Cp < 0x1p100 && Cn < 0x1p100;         // steps stay in a double's range when scaled

    double local_eps = 0;                   // (scaled like f)
    int it = 0;
    // the last step, written to a_sm once every thread has read what it needs for that step
    int step_i = 0, step_j = 0;
    double step_vi = a_sm[0], step_vj = step_vi;
    for (;;) {
        // ---- smallest f over I_up, with its slot -------------------------------------------------------------
        float first_h[CLS];                 // the thread's best
        int first_slot[CLS];
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            float hs[S];
            double v[S];
            int slot[S];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                hs[s] = fmaxf(high_as_float(f[s]), pen_up[c][s]);
                v[s] = with_high(hs[s], f[s]);
                slot[s] = t0 + nth(s);
            }
            // The warp's reduction runs over the high words and needs only their minimum; the exact minimum and its slot
            // are found next to it. Neighbouring slots first: the left operand always holds the lower slots and wins ties.
            const float h = min_of(hs), h_min = warp_min_f32(h);
#pragma unroll
            for (int d = 1; d < S; d <<= 1)
#pragma unroll
                for (int s = 0; s + d < S; s += 2 * d)
                    if (v[s + d] < v[s]) { v[s] = v[s + d]; slot[s] = slot[s + d]; }
            bool winner = h == h_min;
            const unsigned at_min = __ballot_sync(0xffffffffu, winner);
            if ((at_min ^ (at_min - 1)) <= at_min - 1) {        // not one lane: the exact minimum, ties to the lower slot
                unsigned long long key = ordered_key(v[0]);
                int sl = slot[0];
                warp_argmin_u64(key, sl);
                winner = slot[0] == sl;
            }
            if (winner) e1[c][warp] = First{v[0], slot[0], 0};
            first_h[c] = h; first_slot[c] = slot[0];
        }
        solver_barrier<T>();
        double up[CLS];
        int iu[CLS];
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            double v[W];
            int sl[W];
#pragma unroll
            for (int w = 0; w < W; ++w) { const First e = e1[c][w]; v[w] = e.f; sl[w] = e.slot; }
#pragma unroll
            for (int d = 1; d < W; d <<= 1)
#pragma unroll
                for (int w = 0; w + d < W; w += 2 * d)
                    if (v[w + d] < v[w]) { v[w] = v[w + d]; sl[w] = sl[w + d]; }
            up[c] = v[0]; iu[c] = min(sl[0], ws - 1);           // (an empty list)
        }
        float kI[CLS][S], kd_i[CLS];
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            kd_i[c] = ky_sm[iu[c]].x;
            read_row(iu[c], kI[c]);
        }
#pragma unroll
        for (int s = 0; s < S; s += V) {
            if constexpr (V == 4) {
                *(double2 *) (f_sm + t0 + nth(s)) = make_double2(f[s], f[s + 1]);
                *(double2 *) (f_sm + t0 + nth(s + 2)) = make_double2(f[s + 2], f[s + 3]);
            } else f_sm[t0 + nth(s)] = f[s];
        }
        if (tid == 64) { a_sm[step_i] = step_vi; a_sm[step_j] = step_vj; }
        if (AHEAD) {
            best[0][tid] = make_float2(first_h[0], __int_as_float(first_slot[0]));
            if (tid == 96) *(volatile int *) &window[0] = it + 1;
        }
        // the largest f over I_low: high words, clamped to -FAR_POS outside
        float low_h[S], low_most[2] = {-FAR_POS, -FAR_POS};
#pragma unroll
        for (int s = 0; s < S; ++s) low_h[s] = fminf(high_as_float(f[s]), pen_low[s]);
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            float m[S];
#pragma unroll
            for (int s = 0; s < S; ++s) m[s] = !NU || pos[s] == (c == 0) ? low_h[s] : -FAR_POS;
            low_most[c] = warp_max_f32(max_of(m));
        }

        // ---- second-order choice of j ------------------------------------------------------------------------
        // b in FP32, truncated, straight from the double's bits (zero below 2^-126 and outside I_low; the gap bounds it above).
        // A curvature of zero (below 2^-126) has the reciprocal infinity: the value is beyond what is accepted below, whatever b
        // is. A negative one gives a negative value, which counts as zero like that of no candidate: it is chosen only where all
        // values are so, and then in FP64. So does 0 times infinity, slot i itself (the maximum drops a NaN; NaN in a kernel value
        // is found by k_most).
        float q[S], k_most;
        {
            float m[S];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const bool second = NU && !pos[s];
                const float k = second ? kI[CLS - 1][s] : kI[0][s];
                const double b = with_high(low_h[s], f[s]) - (second ? up[CLS - 1] : up[0]);
                const float b32 = __int_as_float(__funnelshift_l((unsigned) __double2loint(b), (unsigned) max(__double2hiint(b), 0), 3));
                const float a32 = fmaf(-2.0f, k, (second ? kd_i[CLS - 1] : kd_i[0]) + kd[s]);
                float r;
                asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a32));
                q[s] = fmaxf(mul_ftz(mul_ftz(b32, r), b32), 0.0f);
                m[s] = k;
            }
            k_most = max_abs3(max_abs_of(m), kd_most, kd_most);
            q[0] = k_most < 1e30f ? q[0] : INFINITY;
        }
        float q2[S];
        int qs[S];
        const float best_w = warp_max_f32(max_of(q));
#pragma unroll
        for (int s = 0; s < S; ++s) { q2[s] = 0.0f; qs[s] = t0 + nth(s); }
#pragma unroll
        for (int d = 1; d < S; d <<= 1)
#pragma unroll
            for (int s = 0; s + d < S; s += 2 * d) {
                q2[s] = d == 1 ? fminf(q[s], q[s + d]) : max3(fminf(q[s], q[s + d]), q2[s], q2[s + d]);
                qs[s] = q[s + d] > q[s] ? qs[s + d] : qs[s];
                q[s] = fmaxf(q[s], q[s + d]);
            }
        {
            const float thr = best_w * (1.0f - 8e-6f);
            const unsigned near = __ballot_sync(0xffffffffu, q[0] >= thr), nears = __ballot_sync(0xffffffffu, q2[0] >= thr);
            if (q[0] == best_w)
                e2[warp] = Second{best_w, (near & (near - 1)) | nears ? qs[0] | TIED : qs[0], {low_most[0], low_most[1]}};
        }
        solver_barrier<T>();
        int j;
        float most[W], next[W], low[CLS];
        double dI[S];
        {
            int sl[W];
            float lw[2][W];
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const Second e = e2[w];
                most[w] = e.best; sl[w] = e.slot; lw[0][w] = e.low[0]; lw[1][w] = e.low[1];
                next[w] = 0;
            }
#pragma unroll
            for (int s = 0; s < S; ++s) dI[s] = NU ? 0.0 : widened(kI[0][s]);
#pragma unroll
            for (int d = 1; d < W; d <<= 1)
#pragma unroll
                for (int w = 0; w + d < W; w += 2 * d) {
                    next[w] = d == 1 ? fminf(most[w], most[w + d]) : max3(fminf(most[w], most[w + d]), next[w], next[w + d]);
                    sl[w] = most[w + d] > most[w] ? sl[w + d] : sl[w];
                    most[w] = fmaxf(most[w], most[w + d]);
                }
            j = min(sl[0] & SLOT_MASK, ws - 1);
            if (sl[0] & TIED) next[0] = most[0];
#pragma unroll
            for (int c = 0; c < CLS; ++c) low[c] = max_of(lw[c]);
        }
        // what the step needs of i and j; read before j is certain
        float kJ[S], kij;
        float2 kyj;
        double fj, aj, ai;
        int yi;
        auto read_step = [&] {
            kyj = ky_sm[j];
            fj = f_sm[j];
            aj = a_sm[j];
            const int i = NU && __float_as_int(kyj.y) < 0 ? iu[CLS - 1] : iu[0];
            kij = __ldg(kww + i * ws + j);          // row i has just been read
            read_row(j, kJ);
            ai = a_sm[i];
            yi = __float_as_int(ky_sm[i].y);
        };
        read_step();
        if (AHEAD) {
            best[1][tid] = make_float2(q[0], __int_as_float(qs[0]));
            if (tid == 96) *(volatile int *) &window[1] = it + 1;
        }
        double gap = 0;
#pragma unroll
        for (int c = 0; c < CLS; ++c) {
            // the smallest double with this high word
            const int h = __float_as_int(low[c]);
            const double g = __hiloint2double(h, h < 0 ? -1 : 0) - up[c];
            gap = c == 0 ? g : fmax(gap, g);
        }
        // ---- the unusual: first and last iteration, a gap that may be closed, values too close to call in FP32 or out of its
        // range (1e-20 .. 3e7, gap below 2^50)
        const bool ranged = (most[0] > 1e-20f) & (most[0] < 3e7f) & (__double2hiint(gap) < (127 + 50) << 20);
        const float tied = most[0] * (1.0f - 8e-6f);
        const bool called = ranged & (next[0] < tied);
        const bool open = ((unsigned) (it - 1) < (unsigned) max_iter) & (gap >= local_eps);
        if (!(called & open)) {
            if (!open) {
                // the exact gap
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
                    const double first = local_diff * BACK;
                    local_eps = (NU ? fmax(eps, 0.1 * first) : fmax(eps, (double) 0.1f * first)) * DOWN;
                    if (tid == 0) diff[0] = first;
                }
                if (it > max_iter || local_diff < local_eps) break;
            }
            if (!called) {
                // the same values in FP64, ties to the lower slot; of a thread with one value that is close enough, only that
                double e_most[CLS];
                int sl[CLS];
                unsigned long long key[CLS];
#pragma unroll
                for (int c = 0; c < CLS; ++c) { e_most[c] = -INFINITY; sl[c] = NO_SLOT; }
                auto weigh = [&](int slot, double fs, float kds, float k, bool second) {
                    const double b = (-(second ? up[CLS - 1] : up[0]) + fs) * BACK;
                    const float kdi = second ? kd_i[CLS - 1] : kd_i[0];
                    const double a = NU ? (double) (kdi + kds - 2 * k) : (double) (kdi + kds) - 2.0 * (double) k;
                    const double e = b * b * reciprocal(a);
#pragma unroll
                    for (int c = 0; c < CLS; ++c)
                        if (b > 0 && second == (c > 0) && e > e_most[c]) { e_most[c] = e; sl[c] = slot; }
                };
                if (!ranged || q2[0] >= tied) {
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        const bool second = NU && !pos[s];
                        if (pen_low[s] > 0) weigh(t0 + nth(s), f[s], kd[s], second ? kI[CLS - 1][s] : kI[0][s], second);
                    }
                } else if (q[0] >= tied) {
                    const float2 ky = ky_sm[qs[0]];
                    const bool second = NU && __float_as_int(ky.y) < 0;
                    weigh(qs[0], f_sm[qs[0]], ky.x, __ldg(kww + (second ? iu[CLS - 1] : iu[0]) * ws + qs[0]), second);
                }
#pragma unroll
                for (int c = 0; c < CLS; ++c) {
                    key[c] = ordered_key(-e_most[c]);
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
                read_step();
            }
        }
        // ---- step, repeated by every thread ------------------------------------------------------------------
        const int yj = __float_as_int(kyj.y);
        const bool second = NU && yj < 0;
        const int i = second ? iu[CLS - 1] : iu[0];
        const double ci = yi > 0 ? Cp : Cn, cj = yj > 0 ? Cp : Cn;
        const double b = (-(second ? up[CLS - 1] : up[0]) + fj) * BACK;
        const float kdi = second ? kd_i[CLS - 1] : kd_i[0];
        const double a = NU ? (double) (kdi + kyj.x - 2 * kij) : (double) (kdi + kyj.x) - 2.0 * (double) kij;
        // b / a by Markstein's method: a reciprocal of most of the digits, the quotient corrected by its remainder
        double r;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
        r = fma(r, fma(-a, r, 1.0), r);
        double l = b * r;
        l = fma(fma(-a, l, b), r, l);
        const double room_i = yi > 0 ? Cp - ai : ai, room_j = yj > 0 ? aj : Cn - aj;
        const double room = room_j < room_i ? room_j : room_i;
        l = room < l ? room : l;
        double d[S];
        float m[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            d[s] = NU ? widened(kJ[s] - (second ? kI[CLS - 1][s] : kI[0][s])) : widened(kJ[s]) - dI[s];
            m[s] = NU ? kJ[s] - (second ? kI[CLS - 1][s] : kI[0][s]) : kJ[s];
        }
        const float k_all = NU ? max_abs_of(m) : max_abs3(max_abs_of(m), k_most, k_most);
        const bool usual = ((unsigned) (__double2hiint(a) - 0x03000000) < 0x79000000u) & mild & (k_all < INFINITY);
        double g[S];
#pragma unroll
        for (int s = 0; s < S; ++s) g[s] = fma(-l, d[s], f[s]);
        if (!usual) {           // curvature not positive or at the ends of the range, infinite kernel values, a huge C
            l = fmin(room, b / a);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float k = second ? kI[CLS - 1][s] : kI[0][s];
                g[s] = fma(-l, NU ? (double) (kJ[s] - k) : (double) kJ[s] - (double) k, f[s] * BACK) * DOWN;
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) f[s] = g[s];
        const double step_ai = ai + (yi > 0 ? l : -l), step_aj = aj - (yj > 0 ? l : -l);
        const bool i_up0 = step_ai < ci, i_dn0 = step_ai > 0, j_up0 = step_aj < cj, j_dn0 = step_aj > 0;
        const bool were_free = (ai > 0) & (ai < ci) & (aj > 0) & (aj < cj);
        if (!(were_free & i_up0 & i_dn0 & j_up0 & j_dn0)) {
            const float up_i = in_I_up(step_ai, yi, Cp, Cn) ? -FAR_POS : FAR_POS, up_j = in_I_up(step_aj, yj, Cp, Cn) ? -FAR_POS : FAR_POS;
            const float lo_i = in_I_low(step_ai, yi, Cp, Cn) ? FAR_POS : -FAR_POS, lo_j = in_I_low(step_aj, yj, Cp, Cn) ? FAR_POS : -FAR_POS;
            const int mine_i = i - t0, mine_j = j - t0;
#pragma unroll
            for (int s = 0; s < S; ++s) {
#pragma unroll
                for (int c = 0; c < CLS; ++c) {
                    if (mine_i == nth(s) && (!NU || second == (c > 0))) pen_up[c][s] = up_i;
                    if (mine_j == nth(s) && (!NU || second == (c > 0))) pen_up[c][s] = up_j;
                }
                if (mine_i == nth(s)) pen_low[s] = lo_i;
                if (mine_j == nth(s)) pen_low[s] = lo_j;
            }
        }
        step_i = i; step_j = j; step_vi = step_ai; step_vj = step_aj;
        ++it;
    }
    if (AHEAD && tid == 0) *(volatile int *) &done = 1;
    solver_barrier<T>();            // (the last step's alphas are in a_sm)
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int t = t0 + nth(s);
        if (t < ws) {
            const double a = a_sm[t], a_old = alpha_ws[t];
            alpha_ws[t] = a;
            alpha_diff[t] = -(a - a_old) * __float_as_int(ky_sm[t].y);
            if (alpha_global && ids[t] >= 0) alpha_global[ids[t]] = a;
        }
    }
    if (tid == 0) {
        diff[1] = it;
        if (times) times->local_end = device_ns();
    }
}

}  // namespace tsvm
