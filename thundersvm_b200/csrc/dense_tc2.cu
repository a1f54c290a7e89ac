// Dense kernel rows on tcgen05 with CTA pairs (cta_group::2).
//
// Every operand is held as two planes (row-scaled FP16, or TF32), a product takes three MMAs, and sums are promoted to FP32
// registers every few k slabs. Two CTAs on neighbouring SMs work as one: the pair owns a 256-instance x 256-requested-row tile,
// each CTA holds the planes of ITS 128 instances and of ITS 128 requested rows (half of the B operand), and one thread of the leader CTA issues tcgen05.mma.cta_group::2 (M = 256), which reads
// both CTAs' shared memory and writes both CTAs' tensor memory. Per CTA a k slab is then 64 KB
// instead of 96 KB for the same tensor-core time, and three of them fit the ring instead of two - the
// single-CTA engine was bound by the latency of its one slab in flight, not by any bandwidth.
//
// Roles per CTA (384 threads = 3 warpgroups): warp 0 TMA producer for this CTA's operand halves
// (transaction bytes are reported to the leader's "full" barrier), warp 1 tensor-memory allocation (both
// CTAs) and MMA issue (leader only), warps 2..3 idle (prediction with the test rows on the lanes: warp 2 fetches the columns'
// numbers), warps 4..11 slab promotion + epilogue on this CTA's 128 instances (prediction with the test rows on the lanes and
// one promotion unit: 640 threads, warps 4..19). Warpgroup 0 hands registers to the others (setmaxnreg): the epilogue keeps 128
// sums per thread live, and with the 168 registers a 384-thread CTA is compiled for it spilled a few loop-invariant
// values - their reloads from local memory (the L1 is tiny next to 222 KB of shared memory) cost 9 % of
// the kernel.
// Barriers: full[s] (leader; both CTAs' TMA bytes), empty[s] (per CTA; MMAs that read the stage have
// retired), tfull[a] (per CTA; slab sum complete), tempty[a] (leader; the epilogue warps of both CTAs drained it).
// Cross-CTA signalling uses mbarrier arrives on shared::cluster addresses and one tcgen05.commit per
// destination CTA; every load is addressed to one CTA's shared memory only. Every mbarrier wait is bounded.
#include "tc_common.cuh"

namespace tsvm {

namespace tc2 {
// A k slab is one 128-byte swizzle row per matrix row: 32 TF32 words or 64 FP16 halves, four MMA k-steps
// of 32 bytes either way.
constexpr int BM = 128, BN = 256, BN_HALF = 128, STAGES = 3, K_STEPS = 4;
constexpr uint32_t A_BYTES = BM * 128;               // 16 KB per plane (this CTA's instances)
constexpr uint32_t B_BYTES = BN_HALF * 128;          // 16 KB per plane (this CTA's half of the requested rows)
constexpr uint32_t STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;   // 64 KB per CTA
// Where 256-column blocks of requested rows would leave most SM pairs idle, the blocks are 128, 64 or 32 columns wide
// (block_width): a tile of few columns is done sooner - its stages are smaller, so that up to five of them are in
// flight, and its epilogue is shorter.
constexpr int MAX_STAGES = 5, MIN_WIDTH = 32;
// Warpgroup 0 holds the TMA producer (warp 0), the MMA issuer (warp 1) and two idle warps and gives most of its
// registers back; the other two warpgroups are the promotion / epilogue warps and take them: two warps per tensor-memory
// lane quarter, 128 columns = 128 sums per thread. (Four warps per quarter with 64 sums each changed nothing on the
// 400,000 x 2,000 launch, 1.90 against 1.88 ms: it waits for the tensor pipe, not for its epilogue.)
constexpr int EPI_WARPS = 8, EPI_WARP0 = 4, THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
constexpr int COLS_PER_THREAD = BN / (EPI_WARPS / 4);
// Registers can only move inside the CTA: what the epilogue warps take (setmaxnreg.inc blocks until it is there)
// must have been given back by the control warps, counted from the per-thread figure the kernel is compiled and
// launched with (168: the largest multiple of 8 with which 384 threads fit 65,536 registers).
constexpr int REGS_LAUNCH = 168, REGS_CONTROL = 56, REGS_EPILOGUE = 224;
static_assert(128 * REGS_CONTROL + 32 * EPI_WARPS * REGS_EPILOGUE <= THREADS * REGS_LAUNCH,
              "the epilogue warps would wait for registers that nobody releases");
static_assert(THREADS * REGS_LAUNCH <= 65536, "register file of an SM");
// Prediction with the test rows on the lanes. Where one promotion unit holds all features (ONE_UNIT) the sums are read from tensor
// memory as the epilogue needs them, and sixteen warps with 64 columns each fit the registers: four per scheduler, which hide
// each other's latencies. Otherwise eight warps keep 128 sums as above.
template <bool ONE_UNIT>
struct Lanes {
    static constexpr int WARPS = ONE_UNIT ? 16 : EPI_WARPS, N_THREADS = 32 * (EPI_WARP0 + WARPS), COLS = BN / (WARPS / 4);
    static constexpr int LAUNCH = ONE_UNIT ? 96 : REGS_LAUNCH, CONTROL = REGS_CONTROL, EPILOGUE = ONE_UNIT ? 104 : REGS_EPILOGUE;
    static_assert(128 * CONTROL + 32 * WARPS * EPILOGUE <= N_THREADS * LAUNCH, "the epilogue warps would wait for registers that nobody releases");
    static_assert(N_THREADS * LAUNCH <= 65536, "register file of an SM");
};
// epilogue staging (see the epilogue): EPI_CHUNK sums of each epilogue thread (eight chunks per thread), and per
// warp the self dots and 1/scale of its requested rows
constexpr int EPI_CHUNK = COLS_PER_THREAD / 8;
constexpr uint32_t EPI_STAGE_BYTES = EPI_CHUNK * EPI_WARPS * 32 * 4;
constexpr uint32_t EPI_CONST_BYTES = EPI_WARPS * 2 * COLS_PER_THREAD * 4;
// prediction form: up to PRED_NC_SMEM coefficients of every epilogue thread's own instance (thread-private columns)
constexpr int PRED_NC_SMEM = 9;
constexpr uint32_t PRED_BYTES = PRED_NC_SMEM * EPI_WARPS * 32 * 4;
// kernel-row form: output row (slot of the caller's row buffer) of every requested row, per epilogue warp
constexpr uint32_t SLOT_BYTES = EPI_WARPS * COLS_PER_THREAD * 4;
constexpr uint32_t SMEM_BASE = STAGES * STAGE_BYTES + 1024 + 256 + EPI_STAGE_BYTES + EPI_CONST_BYTES;
constexpr uint32_t SMEM_BYTES = SMEM_BASE + SLOT_BYTES;
constexpr uint32_t SMEM_BYTES_PREDICT = SMEM_BASE + PRED_BYTES;
// prediction, rows on the lanes: what the epilogue needs of a block's support vectors, COL_ROWS numbers each, twice
constexpr int COL_ROWS = 3 + PRED_NC_SMEM;
constexpr uint32_t COL_BYTES = COL_ROWS * BN * 4;
constexpr uint32_t SMEM_BYTES_LANES = STAGES * STAGE_BYTES + 1024 + 256 + 2 * COL_BYTES;
static_assert(SMEM_BYTES_LANES <= 227 * 1024, "prediction form, rows on the lanes, does not fit the shared memory of an SM");
static_assert(SMEM_BYTES <= 227 * 1024, "kernel-row form does not fit the shared memory of an SM");
static_assert(SMEM_BYTES_PREDICT <= 227 * 1024, "prediction form does not fit the shared memory of an SM");
constexpr uint32_t TMEM_COLS = 512;
// D=F32, K-major, M=256 (two CTAs x 128); A=B=TF32 (format 2) or F16 (format 0)
// (the N field, bits 17.., is added per row block: a block's last rows may need fewer than 256 columns)
constexpr uint32_t IDESC_SHAPE = (1u << 4) | ((uint32_t) (256 >> 4) << 24);
constexpr uint32_t IDESC_TF32 = IDESC_SHAPE | (2u << 7) | (2u << 10);
constexpr uint32_t IDESC_F16 = IDESC_SHAPE;
}  // namespace tc2

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA tile load of a CTA pair: data lands in this CTA's shared memory, the bytes are counted on the
// barrier at the given shared::cluster address (the leader's).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(x), "r"(y) : "memory");
}
// idesc_n: the instruction descriptor's N field ((N >> 3) << 17); a row block with few requested rows left
// issues narrower MMAs
template <bool F16>
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate,
                                          uint32_t idesc_n) {
    if constexpr (F16)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(tc2::IDESC_F16 | idesc_n), "r"(accumulate) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(tc2::IDESC_TF32 | idesc_n), "r"(accumulate) : "memory");
}
// arrives on the barrier at a shared::cluster address once all MMAs issued so far have retired
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster) : "memory");
}

// sums [CH * EPI_CHUNK, (CH + 1) * EPI_CHUNK) of the thread -> its private column of the staging block
template <int CH>
__device__ __forceinline__ void stage_chunk(const float (&sum)[tc2::COLS_PER_THREAD], float *priv) {
    static_assert(tc2::COLS_PER_THREAD / tc2::EPI_CHUNK == 8, "the epilogue's switch lists eight chunks");
#pragma unroll
    for (int c = 0; c < tc2::EPI_CHUNK; ++c) priv[c * (tc2::EPI_WARPS * 32)] = sum[CH * tc2::EPI_CHUNK + c];
}

// Prediction form of the kernel (PREDICT = true): the instances are the support vectors, the requested rows
// the test rows, and instead of writing the kernel values the epilogue multiplies them by the support
// vectors' coefficients and adds the sums to the decision values - svm_kernel::sum_kernel_values
// (src/thundersvm/kernel/kernelmatrix_kernel.cu:69-97) folded into the contraction, so that the
// test x SV kernel block never reaches HBM.
struct PredictArgs {
    const double *coef;        // (n_classes - 1) x n_sv, the model's layout (include/thundersvm/model/svmmodel.h:155-164)
    const int *sv_class;       // class of every support vector [n_sv]
    double *dec;               // the sums are added to dec[r * row_stride + pair * pair_stride]
    long long row_stride, pair_stride;
    int n_classes;
    // rows on the lanes: the support vectors' numbers (predict_columns_kernel), rows of cols_ld floats; FORM % 16 rows of coefficients
    const float *cols;
    long long cols_ld;
};
// form of the kernel: rows, prediction with the instances on the lanes, prediction with the test rows on the lanes and
// FORM % 16 coefficients, for any number of features or for those of one promotion unit
enum { FORM_ROWS = 0, FORM_PREDICT = 1, FORM_LANES = 16, FORM_LANES_ONE_UNIT = 32 };
template <int FORM>
using LanesOf = tc2::Lanes<(FORM >= FORM_LANES_ONE_UNIT)>;

// Optional indirections of the kernel-row form, both read on the device so that a caller can decide them
// without a host round trip: the number of requested rows actually wanted (at most the m the launch was
// sized for) and, per requested row, the row of `out` it is written to.
struct RowsExtra {
    const int *m_dev;
    const int *row_slot;
    int width;                      // requested rows per block (set by the launch)
    int hi_only;                    // the low planes of both operands are zero (set by the launch)
    long long *end;                 // device_ns() when the last block left (never taken back), or nullptr
};

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float sum2(unsigned long long v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;                // two FP32 multiply-adds
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ int pair_index(int n_classes, int i, int j) {      // i < j, pairs ordered (0,1),(0,2),...
    return i * (2 * n_classes - i - 1) / 2 + (j - i - 1);
}

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long exp2_2(unsigned long long v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(lo));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(hi));
    return pack2(lo, hi);
}

// Columns (requested rows) of row block nb that the MMAs cover: all 256, or the rows left rounded up to 32
__device__ __forceinline__ int block_columns(int m, int nb, int width) {
    const int left = m - nb * width;
    return left >= width ? width : ((left + 31) & ~31);
}

__device__ __forceinline__ void red_add_if(bool take, double *p, double v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p red.global.add.f64 [%1], %2;\n\t}" ::"r"((int) take), "l"(p), "d"(v) : "memory");
}

// Prediction: the warp's block of kernel values (32 instances x 16 test rows r0 .. r0 + 15, element (c, l) at column
// (l + c / 2) mod 32 of row c) times the instances' NC coefficients (zero beyond the real ones), added to the decision
// values of the pairs. A lane takes two test rows and eight instances; the four lanes of a pair of rows then add up with
// halving exchanges and end with half of the coefficients of one row.
template <int NC, int CHUNK, int LD>
__device__ __forceinline__ void reduce_chunk(const float *block, const float *coef, int cls_own, int cls_lo, int cls_hi, int r0,
                                             int m, const PredictArgs &pa) {
    static_assert(CHUNK == 16, "eight pairs of rows x four groups of instances");
    constexpr int HALF = (NC + 1) / 2;
    const int lane = threadIdx.x & 31, pair = lane & 7, l0 = (lane >> 3) * 8, odd = (lane >> 3) & 1, high = lane >> 4;
    const int r = r0 + 2 * pair + odd, nc = pa.n_classes - 1;
    for (int cl = cls_lo; cl <= cls_hi; ++cl) {
        const unsigned mine = __ballot_sync(0xffffffffu, cls_own == cl);
        float k[2][8];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int u = 0; u < 8; ++u) k[e][u] = block[(2 * pair + e) * LD + ((l0 + u + pair) & 31)];
        if (mine != 0xffffffffu)
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (!((mine >> (l0 + u)) & 1u)) k[0][u] = k[1][u] = 0.0f;
        unsigned long long k2[2][4];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u) k2[e][u] = pack2(k[e][2 * u], k[e][2 * u + 1]);
        float w[NC];
#pragma unroll
        for (int cr = 0; cr < NC; ++cr) {
            const ulonglong2 ca = *reinterpret_cast<const ulonglong2 *>(coef + cr * LD + l0);
            const ulonglong2 cb = *reinterpret_cast<const ulonglong2 *>(coef + cr * LD + l0 + 4);
            float s[2];
#pragma unroll
            for (int e = 0; e < 2; ++e)
                s[e] = sum2(fma2(cb.y, k2[e][3], fma2(cb.x, k2[e][2], fma2(ca.y, k2[e][1], fma2(ca.x, k2[e][0], 0ull)))));
            w[cr] = (odd ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, odd ? s[0] : s[1], 8);
        }
        double total[HALF];
#pragma unroll
        for (int t = 0; t < HALF; ++t) {
            const float lo = w[t], hi = HALF + t < NC ? w[HALF + t < NC ? HALF + t : t] : 0.0f;
            total[t] = (double) ((high ? hi : lo) + __shfl_xor_sync(0xffffffffu, high ? lo : hi, 16));
        }
        // (no branches: the five exchanges, conversions and additions of ten classes overlap)
        const int above = pair_index(pa.n_classes, cl, cl + 1) - cl;           // pairs (cl, cr + 1) for cr >= cl
#pragma unroll
        for (int t = 0; t < HALF; ++t) {
            const int cr = high * HALF + t;
            const int kp = cr < cl ? pair_index(pa.n_classes, cr, cl) : above + cr;
            red_add_if(cr < nc && r < m, pa.dec + r * pa.row_stride + kp * pa.pair_stride, total[t]);
        }
    }
}

// Prediction with the test rows on the lanes (FORM_LANES + NC): a thread holds the products of one test row with up to 128
// support vectors, so that the sum over them needs no other thread. The support vectors' numbers come from shared memory, the
// same word for all lanes: `col`, rows of BN floats - factor and summand of the exponent (RBF: 2 gamma log2 e / scale, -gamma
// log2 e |x|^2; linear: 1 / scale), class, NC coefficients (zero beyond the real ones). 16 columns at a time, two per
// instruction; sums of 32 products in FP32, of more in FP64. At the end of a class the sums go to its pairs.
template <int I>
struct Index {
    static constexpr int value = I;
    __device__ constexpr operator int() const { return I; }
};
// take(g, x): the products of columns 16 g .. 16 g + 15.
template <int EPI, int NC, bool ONE_UNIT, class Take>
__device__ __forceinline__ void sum_columns(Take take, const float *col, int n_cols, float unscale, float row_term, long long r,
                                            bool wanted, const PredictArgs &pa) {
    using namespace tc2;
    const unsigned long long u2 = pack2(unscale, unscale), a2 = pack2(row_term, row_term);
    double total[NC];
    float part[NC];
#pragma unroll
    for (int t = 0; t < NC; ++t) { total[t] = 0; part[t] = 0; }
    int cls = -1;
    const int nc = pa.n_classes - 1;
    auto add_up = [&] {
#pragma unroll
        for (int t = 0; t < NC; ++t) { total[t] += (double) part[t]; part[t] = 0; }
    };
    auto hand_over = [&] {
        if (NC > 1) add_up();
#pragma unroll
        for (int t = 0; t < NC; ++t) {
            const int pair = NC == 1 ? 0 : t < cls ? pair_index(pa.n_classes, t, cls) : pair_index(pa.n_classes, cls, t + 1);
            red_add_if(wanted && t < nc, pa.dec + r * pa.row_stride + pair * pa.pair_stride, total[t]);
            total[t] = 0;
        }
    };
    auto group = [&](auto g) {
        float x[16];
        take(g, x);
        const float *at = col + g * 16;
        unsigned long long k[8];
#pragma unroll
        for (int p = 0; p < 8; p += 2) {
            const ulonglong2 f = *reinterpret_cast<const ulonglong2 *>(at + 2 * p);
            k[p] = mul2(pack2(x[2 * p], x[2 * p + 1]), u2);
            k[p + 1] = mul2(pack2(x[2 * p + 2], x[2 * p + 3]), u2);
            if constexpr (EPI == EPI_RBF) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(at + BN + 2 * p);
                k[p] = exp2_2(add2(fma2(k[p], f.x, b.x), a2));
                k[p + 1] = exp2_2(add2(fma2(k[p + 1], f.y, b.y), a2));
            } else {
                k[p] = mul2(k[p], f.x);
                k[p + 1] = mul2(k[p + 1], f.y);
            }
        }
        auto accumulate = [&](const unsigned long long (&v)[8]) {
#pragma unroll
            for (int t = 0; t < NC; ++t) {
                unsigned long long w0 = 0ull, w1 = 0ull;
#pragma unroll
                for (int p = 0; p < 8; p += 2) {
                    const ulonglong2 c = *reinterpret_cast<const ulonglong2 *>(at + (3 + t) * BN + 2 * p);
                    w0 = fma2(c.x, v[p], w0);
                    w1 = fma2(c.y, v[p + 1], w1);
                }
                part[t] += sum2(add2(w0, w1));
            }
        };
        if constexpr (NC == 1) accumulate(k);            // (both classes add to the one pair)
        else {
            const int *own = reinterpret_cast<const int *>(at + 2 * BN);
            const int first = own[0], last = own[15];
            if (first == last) {
                if (cls != first && cls >= 0) hand_over();
                cls = first;
                accumulate(k);
            } else
#pragma unroll 1
                for (int c = first; c <= last; ++c) {
                    if (cls != c && cls >= 0) hand_over();
                    cls = c;
                    unsigned long long v[8];
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        float lo, hi;
                        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(k[p]));
                        v[p] = pack2(own[2 * p] == c ? lo : 0.0f, own[2 * p + 1] == c ? hi : 0.0f);
                    }
                    accumulate(v);
                }
        }
    };
    // (n_cols is a multiple of 32)
    if constexpr (ONE_UNIT) {
#pragma unroll 1
        for (int g = 0; g * 16 < n_cols; g += 2) { group(g); group(g + 1); add_up(); }
    } else {                                    // register indices must be constants
        auto two_groups = [&](auto index) {
            constexpr int g = 2 * decltype(index)::value;
            if (g * 16 >= n_cols) return;
            group(Index<g>());
            group(Index<g + 1>());
            add_up();
        };
        two_groups(Index<0>()); two_groups(Index<1>()); two_groups(Index<2>()); two_groups(Index<3>());
    }
    hand_over();
}

template <int EPI, bool F16, int FORM>
__global__ void __launch_bounds__(FORM >= FORM_LANES ? LanesOf<FORM>::N_THREADS : tc2::THREADS, 1)
dense_rows_tc2_kernel(const __grid_constant__ CUtensorMap map_xhi, const __grid_constant__ CUtensorMap map_xlo,
                      const __grid_constant__ CUtensorMap map_whi, const __grid_constant__ CUtensorMap map_wlo,
                      int n, int m_launch, int row_len, const float *__restrict__ sd, const float *__restrict__ sd_rows,
                      const float *__restrict__ x_unscale, const float *__restrict__ w_unscale,
                      KernelFn fn, float *__restrict__ out, long long ld_out, int *__restrict__ status,
                      const PredictArgs pa, const RowsExtra ex) {
    using namespace tc2;
    constexpr bool PREDICT = FORM == FORM_PREDICT, LANES = FORM >= FORM_LANES;
    constexpr bool ONE_UNIT = FORM >= FORM_LANES_ONE_UNIT;
    constexpr int NC = LANES ? FORM % 16 : 1;
    constexpr int WARPS = LANES ? LanesOf<FORM>::WARPS : EPI_WARPS, COLS = LANES ? LanesOf<FORM>::COLS : COLS_PER_THREAD;      // of the epilogue
    // the same value in every thread of the grid: the launch's m, or the smaller count found on the device
    const int m = ex.m_dev ? min(m_launch, max(*ex.m_dev, 0)) : m_launch;
    constexpr int BK = F16 ? 64 : 32;          // elements per k slab
    // k slabs summed in tensor memory before the FP32 promotion (longer units fail the bound on kernel values of 784
    // features in [0, 1])
    constexpr int PROMO = F16 ? 2 : 1;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *ring_ptr = smem_raw + (ring - smem_u32(smem_raw));
    uint64_t *bars = reinterpret_cast<uint64_t *>(ring_ptr + STAGES * STAGE_BYTES);
    const uint32_t full_bar = smem_u32(bars), empty_bar = full_bar + 8 * MAX_STAGES;
    const uint32_t tfull_bar = empty_bar + 8 * MAX_STAGES, tempty_bar = tfull_bar + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * MAX_STAGES + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    // rows on the lanes: two buffers of columns' numbers, filled by warp 2 and read by the epilogue warps
    const uint32_t cfull_bar = smem_u32(bars) + 128, cempty_bar = cfull_bar + 16;
    static_assert(!ONE_UNIT || F16, "one_unit counts halves");
    static_assert((2 * MAX_STAGES + 4) * 8 + 8 <= 128 && 128 + 32 <= 256, "barriers and flags lie side by side");
    const float *colbuf = reinterpret_cast<const float *>(ring_ptr + STAGES * STAGE_BYTES + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const int width = ex.width;
    // One product per value instead of three, and half the bytes, where nothing is left for the low planes: the dense copy of CSR
    // data is made only of values that one FP16 number holds (choose_csr_storage). The products left out are zeros. 16,281 rows
    // against 12,001 x 123: 115 -> 91 us.
    const bool hi_only = F16 && ex.hi_only;
    const uint32_t planes = hi_only ? 1 : 2;
    const uint32_t b_bytes = (uint32_t) width * 64, b_at = planes * A_BYTES, stage_bytes = planes * (A_BYTES + b_bytes);     // half a block's rows of 128 bytes
    const uint32_t n_stages = min((uint32_t) MAX_STAGES, STAGES * STAGE_BYTES / stage_bytes);
    const int pair_tiles = (n + 2 * BM - 1) / (2 * BM), n_blocks = (m + width - 1) / width, k_blocks = (row_len + BK - 1) / BK;
    // Work items are (pair tile, row block) with the row block fastest, so neighbouring clusters stream the
    // same instance slabs at the same time and the second reader finds them in L2.
    // With the test rows on the lanes the tile is the faster one: the support vectors are the larger matrix, and their slabs are
    // read once per launch (200,000 x 2,000 against 100,000 rows: 222 ms the other way round).
    const int n_items = pair_tiles * n_blocks;
    auto tile_of = [&](int item) { return LANES ? item % pair_tiles : item / n_blocks; };
    auto block_of = [&](int item) { return LANES ? item / pair_tiles : item % n_blocks; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar + 8 * a, 1); mbar_init(tempty_bar + 8 * a, 2 * WARPS); }
        if (LANES)
            for (int a = 0; a < 2; ++a) { mbar_init(cfull_bar + 8 * a, 1); mbar_init(cempty_bar + 8 * a, WARPS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();           // both CTAs' barriers are initialised before any remote arrive / TMA
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < EPI_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(LANES ? LanesOf<FORM>::CONTROL : REGS_CONTROL));
    if (warp == 0) {
        // ---------------- TMA producer (both CTAs) ----------------
        if (lane == 0) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (int item = cluster_id; item < n_items && ok; item += n_clusters) {
                    const int pt = tile_of(item), nb = block_of(item);
                    for (int kb = 0; kb < k_blocks; ++kb) {
                        if (!mbar_wait(empty_bar + 8 * stage, phase ^ 1, abort_flag, 1)) { ok = false; break; }
                        const uint32_t base = ring + stage * stage_bytes;
                        const uint32_t leader_full = mapa_u32(full_bar + 8 * stage, 0);
                        if (rank == 0) mbar_expect_tx(full_bar + 8 * stage, 2 * stage_bytes);
                        // this CTA's half of the block's requested rows (a narrow last block has narrow halves)
                        const int xrow = pt * 2 * BM + (int) rank * BM, wrow = nb * width + (int) rank * (block_columns(m, nb, width) >> 1);
                        tma_load_2d_pair(base, &map_xhi, leader_full, kb * BK, xrow);
                        tma_load_2d_pair(base + b_at, &map_whi, leader_full, kb * BK, wrow);
                        if (!hi_only) {
                            tma_load_2d_pair(base + A_BYTES, &map_xlo, leader_full, kb * BK, xrow);
                            tma_load_2d_pair(base + b_at + b_bytes, &map_wlo, leader_full, kb * BK, wrow);
                        }
                        if (++stage == n_stages) { stage = 0; phase ^= 1; }
                    }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA only) ----------------
        if (lane == 0 && rank == 0) {
            uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
            bool ok = true;
            for (int item = cluster_id; item < n_items && ok; item += n_clusters) {
                    const uint32_t idesc_n = (uint32_t) (block_columns(m, block_of(item), width) >> 3) << 17;
                    for (int kb = 0; kb < k_blocks; ++kb) {
                        const bool unit_start = kb % PROMO == 0, unit_end = kb % PROMO == PROMO - 1 || kb == k_blocks - 1;
                        if (unit_start && !mbar_wait(tempty_bar + 8 * acc, acc_phase ^ 1, abort_flag, 2)) { ok = false; break; }
                        if (!mbar_wait(full_bar + 8 * stage, phase, abort_flag, 3)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t d_tmem = tmem_base + acc * BN;
                        const uint32_t base = ring + stage * stage_bytes;
                        if (!hi_only) {
#pragma unroll
                            for (int k = 0; k < K_STEPS; ++k) {
                                const uint32_t koff = k * 32;
                                umma_pair<F16>(d_tmem, smem_desc_sw128(base + A_BYTES + koff),
                                               smem_desc_sw128(base + b_at + koff), k != 0 || !unit_start, idesc_n);
                                umma_pair<F16>(d_tmem, smem_desc_sw128(base + koff),
                                               smem_desc_sw128(base + b_at + b_bytes + koff), 1, idesc_n);
                            }
                        }
#pragma unroll
                        for (int k = 0; k < K_STEPS; ++k) {
                            const uint32_t koff = k * 32;
                            umma_pair<F16>(d_tmem, smem_desc_sw128(base + koff), smem_desc_sw128(base + b_at + koff),
                                           !hi_only || k != 0 || !unit_start, idesc_n);
                        }
                        // stage free / slab complete, signalled in both CTAs
                        umma_commit_pair(mapa_u32(empty_bar + 8 * stage, 0));
                        umma_commit_pair(mapa_u32(empty_bar + 8 * stage, 1));
                        if (++stage == n_stages) { stage = 0; phase ^= 1; }
                        if (unit_end) {
                            umma_commit_pair(mapa_u32(tfull_bar + 8 * acc, 0));
                            umma_commit_pair(mapa_u32(tfull_bar + 8 * acc, 1));
                            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                        }
                    }
            }
        }
    } else if (LANES && warp == 2) {
        // ---------------- the columns' numbers, one block per item (both CTAs, each for itself) ----------------
        if (lane == 0) {
            const uint32_t rows = 3 + NC;
            uint32_t buf = 0, phase = 0;
            for (int item = cluster_id; item < n_items; item += n_clusters) {
                if (!mbar_wait(cempty_bar + 8 * buf, phase ^ 1, abort_flag, 6)) break;
                mbar_expect_tx(cfull_bar + 8 * buf, rows * BN * 4);
                const float *src = pa.cols + (long long) block_of(item) * width;
                for (uint32_t k = 0; k < rows; ++k)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(smem_u32(colbuf) + buf * COL_BYTES + k * (BN * 4)), "l"(src + k * pa.cols_ld), "r"((uint32_t) BN * 4),
                                   "r"(cfull_bar + 8 * buf) : "memory");
                if (++buf == 2) { buf = 0; phase ^= 1; }
            }
        }
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(LANES ? LanesOf<FORM>::EPILOGUE : REGS_EPILOGUE));
        // ---------------- slab promotion + epilogue (both CTAs, own 128 instances) ----------------
        const int quarter = warp & 3, half = (warp - EPI_WARP0) >> 2;
        float *priv = reinterpret_cast<float *>(ring_ptr + STAGES * STAGE_BYTES + 256) + (warp - EPI_WARP0) * 32 + lane;
        float *rowc = reinterpret_cast<float *>(ring_ptr + STAGES * STAGE_BYTES + 256 + EPI_STAGE_BYTES) +
                      (warp - EPI_WARP0) * 2 * COLS_PER_THREAD;
        int *slotc = reinterpret_cast<int *>(ring_ptr + STAGES * STAGE_BYTES + 256 + EPI_STAGE_BYTES + EPI_CONST_BYTES) +
                     (warp - EPI_WARP0) * COLS_PER_THREAD;
        // prediction form: the coefficients of the thread's own instance, one thread-private column
        float *coef_priv = reinterpret_cast<float *>(ring_ptr + STAGES * STAGE_BYTES + 256 + EPI_STAGE_BYTES + EPI_CONST_BYTES) +
                           (warp - EPI_WARP0) * 32 + lane;
        const int nc = PREDICT ? pa.n_classes - 1 : 0;
        uint32_t acc = 0, acc_phase = 0, cbuf = 0, cphase = 0;
        bool ok = true;
        for (int item = cluster_id; item < n_items && ok; item += n_clusters) {
            const int pt = tile_of(item), nb = block_of(item);
            const int j = pt * 2 * BM + (int) rank * BM + quarter * 32 + lane;
            const float sdj = j < n ? sd[j] : 0.0f;
            const float uxj = (F16 && j < n) ? x_unscale[j] : 1.0f;
            const int n_cols = block_columns(m, nb, width);
            int cls_own = 0, cls_lo = 0, cls_hi = -1;
            float coef_one = 0.0f;
            if constexpr (PREDICT) {
                // class and coefficients of the thread's own instance (a lane beyond the last instance takes the
                // last one's class; its kernel values are forced to zero)
                cls_own = pa.sv_class[j < n ? j : n - 1];
                if (nc == 1) coef_one = j < n ? (float) pa.coef[j] : 0.0f;
                else if (nc <= PRED_NC_SMEM)
#pragma unroll
                    for (int cr = 0; cr < PRED_NC_SMEM; ++cr)
                        coef_priv[cr * (EPI_WARPS * 32)] = cr < nc && j < n ? (float) pa.coef[(size_t) cr * n + j] : 0.0f;
            }
            {
                // Self dot and 1/scale of this warp's 128 requested rows go to shared memory by asynchronous
                // copies while the k loop runs: with nearly all of the SM's memory configured as shared, the
                // L1 left over does not keep them across the epilogue's stores.
                const int i0 = nb * width + half * COLS;
#pragma unroll
                for (int c = lane; c < COLS_PER_THREAD; c += 32) {
                    if (!LANES && i0 + c < m) {
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(rowc + c)), "l"(sd_rows + i0 + c) : "memory");
                        if constexpr (F16)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(rowc + COLS_PER_THREAD + c)), "l"(w_unscale + i0 + c) : "memory");
                        if constexpr (FORM == FORM_ROWS)
                            if (ex.row_slot)
                                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(slotc + c)), "l"(ex.row_slot + i0 + c) : "memory");
                    }
                }
                float sum[ONE_UNIT ? 1 : COLS];
                if constexpr (!LANES) {
#pragma unroll
                    for (int c = 0; c < COLS; ++c) sum[c] = 0.0f;
                }
                const float row_term = EPI == EPI_RBF ? -fn.gamma * 1.4426950408889634f * sdj : 0.0f;       // (rows on the lanes)
                for (int unit = 0; unit < (k_blocks + PROMO - 1) / PROMO; ++unit) {
                    if (!mbar_wait(tfull_bar + 8 * acc, acc_phase, abort_flag, 4)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + ((uint32_t) (quarter * 32) << 16) + acc * BN + half * COLS;
                    if constexpr (ONE_UNIT) {
                        if (!mbar_wait(cfull_bar + 8 * cbuf, cphase, abort_flag, 5)) { ok = false; break; }
                        const float *col = colbuf + cbuf * (COL_BYTES / 4) + half * COLS;
                        const int cols = min(n_cols - half * COLS, COLS);
                        if (cols > 0)
                            sum_columns<EPI, NC, true>([&](int g, float (&x)[16]) {
                                uint32_t v[16];
                                tmem_ld16(taddr + 16 * g, v);
#pragma unroll
                                for (int c = 0; c < 16; ++c) x[c] = __uint_as_float(v[c]);
                            }, col, cols, uxj, row_term, j, j < n, pa);
                    } else {
#pragma unroll
                    for (int c0 = 0; c0 < COLS; c0 += 32) {
                        if (half * COLS + c0 >= n_cols) break;      // columns the narrow MMAs did not write
                        uint32_t v[32];
                        tmem_ld32(taddr + c0, v);
                        if (LANES && unit == 0) {
#pragma unroll
                            for (int c = 0; c < 32; ++c) sum[c0 + c] = __uint_as_float(v[c]);
                        } else if constexpr (LANES) {
#pragma unroll
                            for (int c = 0; c < 32; c += 2) {
                                const unsigned long long t = add2(pack2(sum[c0 + c], sum[c0 + c + 1]),
                                                                  pack2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])));
                                asm("mov.b64 {%0, %1}, %2;" : "=f"(sum[c0 + c]), "=f"(sum[c0 + c + 1]) : "l"(t));
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < 32; ++c) sum[c0 + c] += __uint_as_float(v[c]);
                        }
                    }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(mapa_u32(tempty_bar + 8 * acc, 0));
                    if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                }
                if (!ok) break;
                if constexpr (LANES) {
                    if constexpr (!ONE_UNIT) {
                        if (!mbar_wait(cfull_bar + 8 * cbuf, cphase, abort_flag, 5)) { ok = false; break; }
                        const float *col = colbuf + cbuf * (COL_BYTES / 4) + half * COLS;
                        const int cols = min(n_cols - half * COLS, COLS);
                        if (cols > 0)
                            sum_columns<EPI, NC, false>([&](auto g, float (&x)[16]) {
#pragma unroll
                                for (int c = 0; c < 16; ++c) x[c] = sum[16 * decltype(g)::value + c];
                            }, col, cols, uxj, row_term, j, j < n, pa);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(cempty_bar + 8 * cbuf);
                    if (++cbuf == 2) { cbuf = 0; cphase ^= 1; }
                    continue;
                } else {
                // The sums live in registers, so a loop over them has to be fully unrolled; with the kernel
                // function in its body that is 128 copies of it, and the instruction fetch of such an
                // epilogue cost several times its arithmetic. Instead the sums pass 32 at a time through a
                // thread-private column of shared memory (no synchronisation: every thread reads back only
                // what it wrote), 16 at a time, and a short rolled loop applies the kernel function and stores.
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
                // prediction form, RBF: K = 2^(A_i + B_j + S_i * dot) with per-test-row constants A_i, S_i (they
                // replace the row's self dot and 1/scale in rowc) and the own instance's B_j: four instructions
                // per kernel value. The exponent is formed in FP32 without the residual correction the stored
                // kernel rows use (relative error up to |exponent| * 2^-23), which decision values do not need.
                float pred_b = 0.0f;
                if constexpr (PREDICT && EPI == EPI_RBF) {
                    constexpr float LOG2E = 1.4426950408889634f;
                    cls_lo = __reduce_min_sync(0xffffffffu, cls_own);
                    cls_hi = __reduce_max_sync(0xffffffffu, cls_own);
                    pred_b = -fn.gamma * LOG2E * sdj;
#pragma unroll
                    for (int c = lane; c < COLS_PER_THREAD; c += 32) {
                        const float sd_i = rowc[c];
                        const float uw_i = F16 ? rowc[COLS_PER_THREAD + c] : 1.0f;
                        rowc[c] = -fn.gamma * LOG2E * sd_i;
                        rowc[COLS_PER_THREAD + c] = 2.0f * fn.gamma * LOG2E * uw_i;
                    }
                    __syncwarp();
                } else if constexpr (PREDICT) {
                    cls_lo = __reduce_min_sync(0xffffffffu, cls_own);
                    cls_hi = __reduce_max_sync(0xffffffffu, cls_own);
                }
                // the own instance's kernel values with test rows cbase .. cbase + 15, whose sums are in `priv`
                auto values = [&](int cbase, float *kv) {
                    if constexpr (EPI == EPI_RBF) {
                        float a_i[EPI_CHUNK], s_i[EPI_CHUNK];
#pragma unroll
                        for (int c4 = 0; c4 < EPI_CHUNK; c4 += 4) {
                            const float4 av = *reinterpret_cast<const float4 *>(rowc + cbase + c4);
                            const float4 sv = *reinterpret_cast<const float4 *>(rowc + COLS_PER_THREAD + cbase + c4);
                            a_i[c4] = av.x; a_i[c4 + 1] = av.y; a_i[c4 + 2] = av.z; a_i[c4 + 3] = av.w;
                            s_i[c4] = sv.x; s_i[c4 + 1] = sv.y; s_i[c4 + 2] = sv.z; s_i[c4 + 3] = sv.w;
                        }
#pragma unroll
                        for (int c = 0; c < EPI_CHUNK; ++c) {
                            float dot = priv[c * (EPI_WARPS * 32)];
                            if constexpr (F16) dot *= uxj;
                            const float arg = fmaf(dot, s_i[c], a_i[c]) + pred_b;
                            float e;
                            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(arg));
                            kv[c] = j < n ? e : 0.0f;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < EPI_CHUNK; ++c) {
                            float dot = priv[c * (EPI_WARPS * 32)];
                            if constexpr (F16) dot = dot * uxj * rowc[COLS_PER_THREAD + cbase + c];
                            kv[c] = j < n ? epilogue_value<EPI>(fn, dot, rowc[cbase + c], sdj) : 0.0f;
                        }
                    }
                };
                if constexpr (PREDICT) if (nc == 1) {
                    // One coefficient per instance: 32 columns at a time, every value times the instance's coefficient and
                    // then added up over the 32 lanes with exchanges that halve the number of live columns per step (16 + 8
                    // + 4 + 2 + 1 shuffles); lane c ends with column c and adds the warp's sum to the row's place. No
                    // exchange between warps. What bounds it is the chain of the steps, with two such warps per scheduler,
                    // so that 32 columns per chain beat 16: 12,001 x 123 per 4,096 rows 87 -> 64 us, 200,000 x 2,000 7.45 -> 7.3 ms.
                    static_assert(EPI_CHUNK == 16 && COLS_PER_THREAD == 128, "four groups of two chunks");
#pragma unroll 1
                    for (int group = 0; group < COLS_PER_THREAD / 32; ++group) {
                        if (half * COLS_PER_THREAD + group * 32 >= n_cols) break;
                        float kv[32];
                        switch (group) {
                            case 0: stage_chunk<0>(sum, priv); break;
                            case 1: stage_chunk<2>(sum, priv); break;
                            case 2: stage_chunk<4>(sum, priv); break;
                            default: stage_chunk<6>(sum, priv); break;
                        }
                        values(group * 32, kv);
                        switch (group) {
                            case 0: stage_chunk<1>(sum, priv); break;
                            case 1: stage_chunk<3>(sum, priv); break;
                            case 2: stage_chunk<5>(sum, priv); break;
                            default: stage_chunk<7>(sum, priv); break;
                        }
                        values(group * 32 + 16, kv + 16);
                        // (both classes add to the one pair; a lane beyond the last instance has coefficient 0)
                        float w[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const bool upper = (lane & 16) != 0;
                            const float send = coef_one * (upper ? kv[c] : kv[c + 16]);
                            w[c] = fmaf(coef_one, upper ? kv[c + 16] : kv[c], __shfl_xor_sync(0xffffffffu, send, 16));
                        }
#pragma unroll
                        for (int n_left = 8; n_left >= 1; n_left >>= 1)
#pragma unroll
                            for (int c = 0; c < n_left; ++c) {
                                const bool upper = (lane & n_left) != 0;
                                const float send = upper ? w[c] : w[c + n_left];
                                w[c] = (upper ? w[c + n_left] : w[c]) + __shfl_xor_sync(0xffffffffu, send, n_left);
                            }
                        const int r = i0 + group * 32 + lane;
                        if (r < m) atomicAdd(pa.dec + r, (double) w[0]);
                    }
                    __syncwarp();          // the next item's copies overwrite rowc
                    continue;
                }
#pragma unroll 1
                for (int ch = 0; ch < COLS_PER_THREAD / EPI_CHUNK; ++ch) {
                    if (half * COLS_PER_THREAD + ch * EPI_CHUNK >= n_cols) break;
                    switch (ch) {           // register indices must be constants: one short case per chunk
                        case 0: stage_chunk<0>(sum, priv); break;
                        case 1: stage_chunk<1>(sum, priv); break;
                        case 2: stage_chunk<2>(sum, priv); break;
                        case 3: stage_chunk<3>(sum, priv); break;
                        case 4: stage_chunk<4>(sum, priv); break;
                        case 5: stage_chunk<5>(sum, priv); break;
                        case 6: stage_chunk<6>(sum, priv); break;
                        default: stage_chunk<7>(sum, priv); break;
                    }
                    const int cbase = ch * EPI_CHUNK;
                    if constexpr (!PREDICT) {
                        if (j < n) {
                            const int lim = m - (i0 + cbase) < EPI_CHUNK ? m - (i0 + cbase) : EPI_CHUNK;
                            if (!ex.row_slot) {
                                float *o = out + (size_t) (i0 + cbase) * ld_out + j;
#pragma unroll 8
                                for (int c = 0; c < lim; ++c) {
                                    float dot = priv[c * (EPI_WARPS * 32)];
                                    if constexpr (F16) dot = dot * uxj * rowc[COLS_PER_THREAD + cbase + c];
                                    o[(size_t) c * ld_out] = epilogue_value<EPI>(fn, dot, rowc[cbase + c], sdj);
                                }
                            } else {
#pragma unroll 8
                                for (int c = 0; c < lim; ++c) {
                                    float dot = priv[c * (EPI_WARPS * 32)];
                                    if constexpr (F16) dot = dot * uxj * rowc[COLS_PER_THREAD + cbase + c];
                                    out[(size_t) slotc[cbase + c] * ld_out + j] = epilogue_value<EPI>(fn, dot, rowc[cbase + c], sdj);
                                }
                            }
                        }
                    } else {
                        // Several coefficients per instance: the sums of the warp's 32 instances for the chunk's 16 test
                        // rows, as above but once per coefficient where shared memory does not hold them all.
                        float kv[EPI_CHUNK];
                        values(cbase, kv);
                        if (nc > 1 && nc <= PRED_NC_SMEM) {
                            // Several coefficients per instance: the butterfly below would repeat its 31 shuffles for
                            // each of them. Instead the warp's 32 x 16 kernel values go back to shared memory and a lane
                            // takes two columns (test rows) and eight instances (reduce_chunk). Element (c, l) of the block
                            // lies at column (l + c / 2) mod 32, so that stores and reads meet no bank twice. What bounds it
                            // is the chain of these steps, with two such warps per scheduler. Ten classes, 8,003 x 784, per
                            // 4,096 rows: 290 us with the butterfly, 247 with one column and 16 instances per lane (36
                            // instead of 18 reads of coefficients, each as long as four stores), 189 with two, 177 with a
                            // fixed number of coefficients, 173 without branches around the additions, 157 with the
                            // additions side by side.
                            float *block = priv - lane;
                            const float *cf_block = coef_priv - lane;
                            __syncwarp();                    // everyone has read its own sums
#pragma unroll
                            for (int c = 0; c < EPI_CHUNK; ++c) block[c * (EPI_WARPS * 32) + ((lane + c / 2) & 31)] = kv[c];
                            __syncwarp();
                            // (coefficients beyond the real ones are zero: a fixed number keeps the reads in flight together)
                            if (nc <= 3)
                                reduce_chunk<3, EPI_CHUNK, EPI_WARPS * 32>(block, cf_block, cls_own, cls_lo, cls_hi, i0 + cbase, m, pa);
                            else
                                reduce_chunk<PRED_NC_SMEM, EPI_CHUNK, EPI_WARPS * 32>(block, cf_block, cls_own, cls_lo, cls_hi, i0 + cbase, m, pa);
                            __syncwarp();                    // the next chunk's sums overwrite the block
                            continue;
                        }
                        // column of the chunk this lane ends up with: lane bit 16 >> s selects the upper half of step s
                        int col = 0;
#pragma unroll
                        for (int st = 0, hn = EPI_CHUNK / 2; hn >= 1; ++st, hn >>= 1) col += ((lane >> (4 - st)) & 1) * hn;
                        constexpr int REST = 32 / EPI_CHUNK;             // lanes that hold the same column afterwards
                        const int r = i0 + cbase + col;
                        for (int cl = cls_lo; cl <= cls_hi; ++cl)
                            for (int cr = 0; cr < nc; ++cr) {
                                float cf = j < n ? (float) pa.coef[(size_t) cr * n + j] : 0.0f;
                                if (cls_own != cl) cf = 0.0f;
                                float w[EPI_CHUNK];
#pragma unroll
                                for (int c = 0; c < EPI_CHUNK; ++c) w[c] = cf * kv[c];
#pragma unroll
                                for (int st = 0, half_n = EPI_CHUNK / 2; half_n >= 1; ++st, half_n >>= 1) {
                                    const int bit = 16 >> st;                          // lane bit 4, 3, 2, ...
                                    const bool upper = (lane & bit) != 0;
#pragma unroll
                                    for (int c = 0; c < half_n; ++c) {
                                        const float send = upper ? w[c] : w[c + half_n];
                                        const float keep = upper ? w[c + half_n] : w[c];
                                        w[c] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                                    }
                                }
                                float total = w[0];
#pragma unroll
                                for (int o = REST >> 1; o >= 1; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
                                if ((lane & (REST - 1)) == 0 && r < m && total != 0.0f) {
                                    const int k = cr < cl ? pair_index(pa.n_classes, cr, cl) : pair_index(pa.n_classes, cl, cr + 1);
                                    atomicAdd(pa.dec + r * pa.row_stride + k * pa.pair_stride, (double) total);
                                }
                            }
                    }
                }
                __syncwarp();          // the next item's copies overwrite rowc
                }
            }
        }
    }

    if (*abort_flag) {
        const long long t0 = device_ns();
        while (device_ns() - t0 < 1000000ll) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();           // neither CTA leaves while its partner may still signal it or read its memory
    tc_fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    if (threadIdx.x == 0 && ex.end) atomicMax(ex.end, device_ns());
    if (threadIdx.x == 0 && *abort_flag) *(volatile int *) status = *abort_flag;      // (may be a word of pinned host memory)
}

tsvm_status make_map(CUtensorMap *map, const void *ptr, int rows, int row_len, long long ld, int box_rows,
                     bool f16);   // dense_tc.cu

// Columns per block: halved while every tile still gets an SM pair of its own, i.e. as long as it costs no second round. A
// tile takes 5 us, 0.73 (32 columns) to 0.87 us per k slab and 1 to 5 us of epilogue. 512 requested rows of 1,024 x 64 /
// 784 / 2,000: 11.6 / 22.3 / 38.8 -> 6.5 / 15.6 / 29.8 us; predicting 100 rows with 1,000 x 100 70 -> 64 us, 300 with 2,000
// x 2,000 104 -> 93 us.
static int block_width(int pair_tiles, int m, int avail) {
    int width = tc2::BN;
    while (width > tc2::MIN_WIDTH && (long long) pair_tiles * ceil_div(m, width / 2) <= avail) width /= 2;
    return width;
}

template <int EPI, bool F16, int FORM>
static tsvm_status launch_pair_kernel(tsvm_km *km, const InstancePlanes &X, const RowPlanes &W, int m, float *out,
                                      long long ld_out, const PredictArgs &pa, const RowsExtra &ex_in, cudaStream_t st) {
    auto kernel = dense_rows_tc2_kernel<EPI, F16, FORM>;
    constexpr uint32_t smem_bytes = FORM >= FORM_LANES ? tc2::SMEM_BYTES_LANES
                                  : FORM == FORM_PREDICT ? tc2::SMEM_BYTES_PREDICT : tc2::SMEM_BYTES;
    constexpr int threads = FORM >= FORM_LANES ? LanesOf<FORM>::N_THREADS : tc2::THREADS;
    static int clusters_of_device[MAX_DEVICES] = {0};      // per instantiation and per device ordinal
    int dev = 0;
    TSVM_CUDA(cudaGetDevice(&dev));
    int &max_clusters = clusters_of_device[dev & (MAX_DEVICES - 1)];
    if (!max_clusters) {
        int sms = 0;
        TSVM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        TSVM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem_bytes));
        cudaLaunchConfig_t probe = {};
        cudaLaunchAttribute pattr[1];
        pattr[0].id = cudaLaunchAttributeClusterDimension;
        pattr[0].val.clusterDim.x = 2; pattr[0].val.clusterDim.y = 1; pattr[0].val.clusterDim.z = 1;
        probe.gridDim = dim3(sms & ~1); probe.blockDim = dim3(threads); probe.dynamicSmemBytes = smem_bytes;
        probe.attrs = pattr; probe.numAttrs = 1;
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, kernel, &probe) != cudaSuccess || nc < 1) {
            cudaGetLastError();
            nc = sms / 2;
        }
        max_clusters = nc;
    }
    CUtensorMap mxh, mxl, mwh, mwl;
    const int len = km->plane_ld;
    TSVM_TRY(make_map(&mxh, X.hi, X.n, len, len, tc2::BM, F16));
    TSVM_TRY(make_map(&mxl, X.lo, X.n, len, len, tc2::BM, F16));
    int avail = max_clusters - km->reserve_clusters;     // SM pairs left free for a concurrent stream
    if (avail < 1) avail = 1;
    RowsExtra ex = ex_in;
    ex.hi_only = km->from_csr;
    ex.width = km->whole_blocks ? tc2::BN : block_width(ceil_div(X.n, 2 * tc2::BM), m, avail);
    TSVM_TRY(make_map(&mwh, W.hi, m, len, len, ex.width / 2, F16));
    TSVM_TRY(make_map(&mwl, W.lo, m, len, len, ex.width / 2, F16));
    const int n_items = ceil_div(X.n, 2 * tc2::BM) * ceil_div(m, ex.width);
    const int clusters = n_items < avail ? n_items : avail;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2 * clusters); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 1;
    TSVM_CUDA(cudaLaunchKernelEx(&cfg, kernel, mxh, mxl, mwh, mwl, X.n, m, len, X.sd, W.sd, X.unscale, W.unscale,
                                 km->fn, out, ld_out, FORM != FORM_ROWS ? km->status_host : km->status_dev, pa, ex));
    count_launch();
    return TSVM_OK;
}

template <int FORM>
static tsvm_status launch_pair_any(tsvm_km *km, const InstancePlanes &X, const RowPlanes &W, int m, float *out,
                                   long long ld_out, const PredictArgs &pa, const RowsExtra &ex, cudaStream_t st) {
    TSVM_REQUIRE(km->plane_kind == 1 || km->plane_kind == 2, "tensor engine: operand planes are not built");
    const int epi = epilogue_kind(km->fn);
    if (km->plane_kind == 2) {
        if (epi == EPI_RBF) return launch_pair_kernel<EPI_RBF, true, FORM>(km, X, W, m, out, ld_out, pa, ex, st);
        if (epi == EPI_LINEAR) return launch_pair_kernel<EPI_LINEAR, true, FORM>(km, X, W, m, out, ld_out, pa, ex, st);
        return launch_pair_kernel<EPI_GENERIC, true, FORM>(km, X, W, m, out, ld_out, pa, ex, st);
    }
    if (epi == EPI_RBF) return launch_pair_kernel<EPI_RBF, false, FORM>(km, X, W, m, out, ld_out, pa, ex, st);
    if (epi == EPI_LINEAR) return launch_pair_kernel<EPI_LINEAR, false, FORM>(km, X, W, m, out, ld_out, pa, ex, st);
    return launch_pair_kernel<EPI_GENERIC, false, FORM>(km, X, W, m, out, ld_out, pa, ex, st);
}

// Kernel values of the m staged requested rows against a set of instances given by its operand planes
// (kind 1 = TF32 words, 2 = row-scaled FP16, the handle's plane kind), self dots and 1/scale.
tsvm_status launch_dense_tc2_planes(tsvm_km *km, const InstancePlanes &X, const RowPlanes &W, int m, float *out,
                                    long long ld_out, cudaStream_t st) {
    return launch_pair_any<FORM_ROWS>(km, X, W, m, out, ld_out, PredictArgs{}, RowsExtra{km->rows_m_dev, km->rows_slot_dev, 0, 0, km->rows_end_dev}, st);
}

// Prediction form: the m staged rows are test rows, the kernel matrix holds the support vectors; adds
// sum_sv coef * K(sv, test row) to dec_dev[r * n_pairs + pair] (preset by the caller) without writing K.
tsvm_status launch_dense_tc2_predict(tsvm_km *km, int m, const double *coef_dev, const int *sv_class_dev,
                                     int n_classes, double *dec_dev, long long row_stride, long long pair_stride, cudaStream_t st) {
    const InstancePlanes all{km->Xhi, km->Xlo, km->self_dot, km->x_unscale, km->n};
    const RowPlanes staged{km->Whi, km->Wlo, km->sd_rows, km->w_unscale};
    const PredictArgs pa{coef_dev, sv_class_dev, dec_dev, row_stride, pair_stride, n_classes, nullptr, 0};
    return launch_pair_any<FORM_PREDICT>(km, all, staged, m, nullptr, 0, pa, RowsExtra{nullptr, nullptr, 0, 0, nullptr}, st);
}

// The same with the test rows on the tensor memory's lanes and the support vectors on its columns. What bounds FORM_PREDICT is
// its epilogue: the sum over the support vectors crosses the lanes of a warp (19 instructions per warp and kernel value with
// two classes, 58 with ten, waiting included); here it stays in a thread, and the support vectors' numbers are the same words
// for all lanes (8 and 44). Kernel times: 16,281 x 12,001 x 123 254 us in four launches -> 115 us in one (91 with one product),
// ten classes, 10,000 x 8,003 x 784 380 us in three -> 323 us in one; whole calls 320 -> 142 and 535 -> 405 us, 100,000 x
// 200,000 x 2,000 184 -> 181 ms (it waits for the tensor pipe). What bounds it now: with 123 features and three products those,
// 2.4 of 2.8 us per tile (with one, see hi_only, the epilogue); with ten classes the epilogue (products alone: 240 of 323 us).
// Sums are no less exact than before: FP32 over four products at a time, FP64 from 32 on; against sums in FP64 the relative
// errors of ten data sets are 0.96 - 1.03 times the former, 1.00 on average.
// The price is a tile of 256 test rows, whole or not. The columns' numbers travel by bulk copies into two buffers (warp 2), so
// that the epilogue's warps need no barrier among themselves.
tsvm_status launch_dense_tc2_predict_lanes(tsvm_km *km, int m, const float *cols, long long cols_ld, int nc_pad, int n_classes,
                                           double *dec_dev, long long row_stride, long long pair_stride, cudaStream_t st) {
    const InstancePlanes rows{km->Whi, km->Wlo, km->sd_rows, km->w_unscale, m};
    const RowPlanes svs{km->Xhi, km->Xlo, km->self_dot, km->x_unscale};
    const PredictArgs pa{nullptr, nullptr, dec_dev, row_stride, pair_stride, n_classes, cols, cols_ld};
    const RowsExtra ex{nullptr, nullptr, 0, 0, nullptr};
    const bool rbf = epilogue_kind(km->fn) == EPI_RBF;
    const bool one_unit = km->plane_ld <= 128;              // two k slabs
#define TSVM_LANES(EPI, NC) \
    (one_unit ? launch_pair_kernel<EPI, true, FORM_LANES_ONE_UNIT + NC>(km, rows, svs, km->n, nullptr, 0, pa, ex, st) \
              : launch_pair_kernel<EPI, true, FORM_LANES + NC>(km, rows, svs, km->n, nullptr, 0, pa, ex, st))
    if (rbf) return nc_pad == 1 ? TSVM_LANES(EPI_RBF, 1) : nc_pad == 3 ? TSVM_LANES(EPI_RBF, 3) : TSVM_LANES(EPI_RBF, 9);
    return nc_pad == 1 ? TSVM_LANES(EPI_LINEAR, 1) : nc_pad == 3 ? TSVM_LANES(EPI_LINEAR, 3) : TSVM_LANES(EPI_LINEAR, 9);
#undef TSVM_LANES
}

// Requested rows = the m rows staged in the handle's scratch.
tsvm_status launch_dense_tc2_on(tsvm_km *km, const InstancePlanes &X, int m, float *out, long long ld_out,
                                cudaStream_t st) {
    const RowPlanes staged{km->Whi, km->Wlo, km->sd_rows, km->w_unscale};
    return launch_dense_tc2_planes(km, X, staged, m, out, ld_out, st);
}

// The same against all instances of the kernel matrix.
tsvm_status launch_dense_tc2(tsvm_km *km, int m, float *out, long long ld_out, cudaStream_t st) {
    const InstancePlanes all{km->Xhi, km->Xlo, km->self_dot, km->x_unscale, km->n};
    return launch_dense_tc2_on(km, all, m, out, ld_out, st);
}

}  // namespace tsvm
