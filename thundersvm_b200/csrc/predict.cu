// Prediction: decision values of a batch of test instances against the support vectors.
// Reference behaviour: SvmModel::predict_dec_values (src/thundersvm/model/svmmodel.cpp:74-117),
// svm_kernel::sum_kernel_values (src/thundersvm/kernel/kernelmatrix_kernel.cu:69-97), the vote of
// SVC::predict_label (src/thundersvm/model/svc.cpp:265-289) and the vote-only form
// sum_kernel_values_instant (kernelmatrix_kernel.cu:99-138).
//
// Three paths:
//   * a few test rows (predict_few.cuh): one launch, FP32 dot products on CUDA cores;
//   * dense support vectors of more than 32 features, and CSR ones that the handle also keeps as dense rows
//     (choose_csr_storage) if the test rows qualify too: the test x SV contraction multiplies its kernel values by
//     the coefficients in its epilogue and adds them to the decision values (dense_tc2.cu, prediction forms), so the
//     kernel block is never written; more than LANES_ROWS rows, RBF and linear kernels and up to ten classes: with the
//     test rows on the accumulator's lanes, otherwise with the support vectors on them;
//   * the rest compute the block in slabs of test rows and reduce it with sum_kernel_values_kernel.
#include "common.cuh"
#include "predict_few.cuh"
#include <vector>

namespace tsvm {

// One block per test row. For every class pair (i, j), i < j, in the reference's order:
//   dec = sum_{s in class i} coef[(j-1) n_sv + s] K[s] + sum_{s in class j} coef[i n_sv + s] K[s] - rho[k]
// with double accumulation; K and coef are read with unit stride across the block.
__global__ void __launch_bounds__(256)
sum_kernel_values_kernel(const double *__restrict__ coef, int n_sv, const int *__restrict__ sv_start,
                         const int *__restrict__ sv_count, const double *__restrict__ rho,
                         const float *__restrict__ K, long long ldk, double *__restrict__ dec, int n_classes) {
    __shared__ double part[2][8];
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *kv = K + (size_t) r * ldk;
    const int nb = n_classes * (n_classes - 1) / 2;
    int k = 0;
    for (int i = 0; i < n_classes; ++i)
        for (int j = i + 1; j < n_classes; ++j, ++k) {
            const double *c1 = coef + (size_t) (j - 1) * n_sv + sv_start[i];
            const double *c2 = coef + (size_t) i * n_sv + sv_start[j];
            const float *k1 = kv + sv_start[i], *k2 = kv + sv_start[j];
            const int n1 = sv_count[i], n2 = sv_count[j];
            double s = 0;
            for (int l = tid; l < n1; l += 256) s += c1[l] * (double) k1[l];
            for (int l = tid; l < n2; l += 256) s += c2[l] * (double) k2[l];
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            double *buf = part[k & 1];
            if (lane == 0) buf[warp] = s;
            __syncthreads();
            if (tid == 0) {
                double t = 0;
                for (int w = 0; w < 8; ++w) t += buf[w];
                dec[(size_t) r * nb + k] = t - rho[k];
            }
        }
}

// Three to SLAB_CLASSES classes: the contraction adds to a slab [pair][row], where the rows that a warp adds to at a time lie
// side by side (to [row][pair] every one is a memory sector of its own: ten classes, 8,003 x 784, 173 -> 157 us per
// 4,096 rows). This kernel turns the slab into decision values [row][pair] and / or votes (the first maximum wins).
constexpr int SLAB_CLASSES = 32, SLAB_THREADS = 256;
static bool sums_by_pair(int n_classes) { return n_classes > 2 && n_classes <= SLAB_CLASSES; }
__global__ void __launch_bounds__(SLAB_THREADS)
finish_slab_kernel(const double *__restrict__ slab, long long ld, int m, int n_classes, double *__restrict__ dec,
                   int *__restrict__ labels) {
    __shared__ double tile[32][33];
    __shared__ int votes[SLAB_CLASSES][32];
    __shared__ unsigned char first[SLAB_CLASSES * (SLAB_CLASSES - 1) / 2], second[SLAB_CLASSES * (SLAB_CLASSES - 1) / 2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r0 = blockIdx.x * 32, nb = n_classes * (n_classes - 1) / 2;
    for (int e = tid; e < n_classes * 32; e += SLAB_THREADS) votes[e >> 5][e & 31] = 0;
    for (int e = tid; e < n_classes * n_classes; e += SLAB_THREADS) {
        const int i = e / n_classes, j = e - i * n_classes;
        if (i < j) {
            const int k = i * (2 * n_classes - i - 1) / 2 + (j - i - 1);
            first[k] = i; second[k] = j;
        }
    }
    __syncthreads();
    for (int k0 = 0; k0 < nb; k0 += 32) {
#pragma unroll
        for (int u = 0; u < 32; u += SLAB_THREADS / 32) {
            const int k = k0 + u + warp;
            if (k < nb && r0 + lane < m) {
                const double v = slab[k * ld + r0 + lane];
                if (dec) tile[u + warp][lane] = v;
                if (labels) atomicAdd(&votes[v > 0 ? first[k] : second[k]][lane], 1);
            }
        }
        if (!dec) continue;
        __syncthreads();
        for (int u = warp; u < 32; u += SLAB_THREADS / 32)
            if (r0 + u < m && k0 + lane < nb) dec[(size_t) (r0 + u) * nb + k0 + lane] = tile[lane][u];
        __syncthreads();
    }
    if (!labels) return;
    __syncthreads();
    if (tid < 32 && r0 + tid < m) {
        int best = 0;
        for (int c = 1; c < n_classes; ++c)
            if (votes[c][tid] > votes[best][tid]) best = c;
        labels[r0 + tid] = best;
    }
}

// Class tables from the per-class counts, which travel as a kernel argument (no copy to wait for): start and count of
// every class, class of every support vector.
constexpr int ARG_CLASSES = 512;
struct ClassCounts { int count[ARG_CLASSES]; };
__global__ void class_tables_kernel(const __grid_constant__ ClassCounts cc, int n_classes, int n_sv, int *__restrict__ start,
                                    int *__restrict__ count, int *__restrict__ cls) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    int at = 0;
    for (int c = 0; c < n_classes; ++c) {
        const int n = cc.count[c];
        if (s == c) { start[c] = at; count[c] = n; }
        if (cls && s >= at && s < at + n) cls[s] = c;
        at += n;
    }
}

// What the contraction with the test rows on the lanes needs of every support vector, one row of `ld` floats each (zero beyond
// the last support vector): factor and summand of the kernel function's argument, class, nc_pad coefficients.
constexpr int LANES_CLASSES = 10;
static int lanes_coefficients(int n_classes) { return n_classes == 2 ? 1 : n_classes <= 4 ? 3 : LANES_CLASSES - 1; }
__global__ void predict_columns_kernel(const __grid_constant__ ClassCounts cc, int n_classes, int n_sv, long long ld, int nc_pad,
                                       const double *__restrict__ coef, const float *__restrict__ sd,
                                       const float *__restrict__ unscale, int rbf, float gamma, float *__restrict__ out) {
    const long long s = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ld) return;
    const bool there = s < n_sv;
    int cls = 0;
    for (int c = 0, end = 0; c + 1 < n_classes; ++c) { end += cc.count[c]; cls += s >= end; }
    constexpr float LOG2E = 1.4426950408889634f;
    const float u = there ? unscale[s] : 0.0f;
    out[s] = rbf ? 2.0f * gamma * LOG2E * u : u;
    out[ld + s] = rbf && there ? -gamma * LOG2E * sd[s] : 0.0f;
    out[2 * ld + s] = __int_as_float(cls);
    for (int t = 0; t < nc_pad; ++t) out[(3 + t) * ld + s] = there && t < n_classes - 1 ? (float) coef[(size_t) t * n_sv + s] : 0.0f;
}

// the classes from start offsets in memory (more classes than the argument holds)
__global__ void sv_class_kernel(int *__restrict__ cls, int n_sv, const int *__restrict__ sv_start, int n_classes) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n_sv) return;
    int c = 0;
    while (c + 1 < n_classes && s >= sv_start[c + 1]) ++c;
    cls[s] = c;
}

// votes -> index of the winning class, first maximum wins. One warp per row: the signs of the row's decision values are
// packed into words (coalesced reads), then every lane counts the votes of its classes. 4,096 rows of ten classes: 25 -> 3.5 us
// against one thread per row.
constexpr int VOTE_WARPS = 8, VOTE_WORDS = 256;            // at most 8,192 pairs
__global__ void __launch_bounds__(VOTE_WARPS * 32)
vote_kernel(const double *__restrict__ dec, int m, int n_classes, int *__restrict__ out) {
    __shared__ unsigned sign[VOTE_WARPS][VOTE_WORDS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = blockIdx.x * VOTE_WARPS + warp;
    if (r >= m) return;
    const int nb = n_classes * (n_classes - 1) / 2;
    const double *d = dec + (size_t) r * nb;
    for (int k0 = 0; k0 < nb; k0 += 32) {
        const unsigned w = __ballot_sync(0xffffffffu, k0 + lane < nb && d[k0 + lane] > 0);
        if (lane == 0) sign[warp][k0 >> 5] = w;
    }
    __syncwarp();
    int best = -1;                                          // (votes, class) packed: more votes first, then the lower class
    for (int c = lane; c < n_classes; c += 32) {
        int votes = 0;
        for (int o = 0; o < n_classes; ++o) {
            if (o == c) continue;
            const int i = o < c ? o : c, j = o < c ? c : o;
            const int k = i * (2 * n_classes - i - 1) / 2 + (j - i - 1);
            const unsigned pos = (sign[warp][k >> 5] >> (k & 31)) & 1u;
            votes += o > c ? pos : 1u - pos;
        }
        best = max(best, votes * 256 + (255 - c));
    }
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0) out[r] = 255 - (best & 255);
}

// any number of classes: one thread per row
__global__ void vote_many_kernel(const double *__restrict__ dec, int m, int n_classes, int *__restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    const int nb = n_classes * (n_classes - 1) / 2;
    int best = 0, best_votes = -1;
    for (int c = 0; c < n_classes; ++c) {
        int votes = 0, k = 0;
        for (int i = 0; i < n_classes; ++i)
            for (int j = i + 1; j < n_classes; ++j, ++k) {
                const bool pos = dec[(size_t) r * nb + k] > 0;
                if ((pos && i == c) || (!pos && j == c)) ++votes;
            }
        if (votes > best_votes) { best_votes = votes; best = c; }
    }
    out[r] = best;
}

static tsvm_status launch_vote(const double *dec, int m, int n_classes, int *out, cudaStream_t st) {
    if (n_classes <= 128)
        TSVM_LAUNCH(vote_kernel, ceil_div(m, VOTE_WARPS), VOTE_WARPS * 32, 0, st, dec, m, n_classes, out);
    else TSVM_LAUNCH(vote_many_kernel, ceil_div(m, 128), 128, 0, st, dec, m, n_classes, out);
    return TSVM_OK;
}

}  // namespace tsvm

using namespace tsvm;

// Rows of test instances handled per launch of the fused contraction (the handle's staging scratch grows to hold them): as
// many as leave their operand planes in a quarter of the L2 cache, where every block of support vectors reads them again, and
// at least 4,096; `scratch_pairs` decision values per row that the call keeps for itself may take a sixteenth of the device,
// like the kernel block of the unfused path, or what 16,384 rows need: with more than 128 classes the vote is a thread per row and
// takes as long for 4,096 rows as for these (16,384 rows, 150 classes: 670 ms in four launches, 180 in one). Whole calls with
// 4,096 / 16,384 / as many rows per launch as the planes allow: 60,000 rows against 12,001 x 123 one-hot CSR 630 / 440 / 392 us,
// 100,000 against 3,000 x 60 588 / 317 / 215, 300,000 against 1,000 x 64, three classes, 1,400 - 2,000 / 650 - 820 / 370 - 440, 60,000
// against 2,000 x 100, 20 classes, 3,490 / 2,400 / 2,210, 60 classes 18.6 / 15.4 / 15.2 ms. Half and twice the quarter: 100,000 against
// 3,000 x 60 226 / 214, 40,000 against 40,000 x 2,000 15.1 and 15.6 - 17.1 ms against 14.5 - 15.1.
static int fused_rows(const tsvm_km *km, size_t scratch_pairs) {
    size_t fit = device_l2_bytes() / 4 / (2 * km_plane_row_bytes(km));
    if (fit < 4096) fit = 4096;
    size_t most = device_memory_bytes() / 16 / (sizeof(double) * (scratch_pairs ? scratch_pairs : 1));
    if (most < 16384) most = 16384;
    return (int) ((fit < most ? fit : most) & ~(size_t) 255);
}
// From this number of test rows on the contraction takes them on the lanes of its accumulators (FORM_LANES in dense_tc2.cu): its
// epilogue is the shorter one, but it computes whole tiles of 256 rows. 40,000 x 2,000, both forms: 157 against 166 us with
// 129 rows, 164 / 168 with 192, 176 / 169 with 256, 239 / 230 with 257, 399 / 382 with 800; smaller models differ by less.
static constexpr int LANES_ROWS = 192;

// Decision values of test rows [r0, r0 + mm) into dec (preset here): [row][pair] with pair_stride 1, else [pair][row].
static tsvm_status fused_slab(tsvm_km *km_sv, const double *coef_dev, const int *sv_class, const float *columns, long long columns_ld,
                              const double *rho_dev, int n_classes, long long r0, int mm, const float *T_dev, int dt, int ldt,
                              const float *tval_dev, const int *trow_ptr_dev, const int *tcol_dev, double *dec,
                              long long pair_stride, cudaStream_t st) {
    const int nb = n_classes * (n_classes - 1) / 2;
    const long long total = pair_stride == 1 ? (long long) mm * nb : pair_stride * nb;
    SumPreset preset;
    preset.sums = dec; preset.rho = rho_dev; preset.total = total; preset.pair_stride = pair_stride; preset.n_pairs = nb;
    if (T_dev) TSVM_TRY(km_stage_instances_dense(km_sv, T_dev + (size_t) r0 * ldt, mm, dt, ldt, preset, st));
    else TSVM_TRY(km_stage_instances_csr(km_sv, tval_dev, trow_ptr_dev + r0, tcol_dev, mm, preset, st));
    const long long row_stride = pair_stride == 1 ? nb : 1;
    if (columns)
        return launch_dense_tc2_predict_lanes(km_sv, mm, columns, columns_ld, lanes_coefficients(n_classes), n_classes, dec, row_stride,
                                              pair_stride, st);
    return launch_dense_tc2_predict(km_sv, mm, coef_dev, sv_class, n_classes, dec, row_stride, pair_stride, st);
}

// Few rows: one launch (predict_few.cuh; 62 -> 33 us per call at 8 rows x 3,001 x 100, 104 -> 45 us at 1 x 5,000 x 784 with
// ten classes, 190 -> 42 us at 5 CSR rows x 8,000). *taken: the path was taken and the results are there.
// Where the line lies: eight rows cost one read of the support vectors, which no other path undercuts; more rows cost
// one read (from L2) per eight, so that they pay as long as that stays below the 15 - 20 us that the general path's
// extra launches take - about 1.6e7 features read.
template <int R>
static tsvm_status launch_few(const FewArgs &a, bool csr, cudaStream_t st) {
    const int tiles = ceil_div(a.m, R);
    int bx = ceil_div(a.n_sv, 8), most = 2 * device_sm_count() / tiles;
    if (most < 1) most = 1;
    if (bx > most) bx = most;
    if (csr) {
        const size_t smem = sizeof(float) * FEW_ENTRIES * R + (sizeof(int) + sizeof(short)) * FEW_SLOTS + FewShared<R>::bytes(a.n_pairs);
        TSVM_ONCE_PER_DEVICE(TSVM_CUDA(cudaFuncSetAttribute(predict_few_csr_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)));
        TSVM_LAUNCH(predict_few_csr_kernel<R>, dim3(bx, tiles), FEW_THREADS + 32, smem, st, a);
    } else {
        const size_t smem = sizeof(float) * R * ((a.d + 3) & ~3) + FewShared<R>::bytes(a.n_pairs);
        TSVM_ONCE_PER_DEVICE(TSVM_CUDA(cudaFuncSetAttribute(predict_few_dense_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)));
        TSVM_LAUNCH(predict_few_dense_kernel<R>, dim3(bx, tiles), FEW_THREADS + 32, smem, st, a);
    }
    return TSVM_OK;
}

static tsvm_status predict_few(tsvm_km *km, const double *coef_dev, const int *sv_count_host, const double *rho_dev,
                               int n_classes, int m, const float *T_dev, int dt, int ldt, const float *tval_dev,
                               const int *trow_ptr_dev, const int *tcol_dev, long long tnnz, double *dec_dev, int *labels_dev,
                               cudaStream_t st, bool *taken) {
    *taken = false;
    const bool dense = km->dense && !km->from_csr;      // few rows: the entries are read once, and there are fewer of them
    const int R = m == 1 ? 1 : (m == 2 ? 2 : (m <= 4 ? 4 : 8)), tiles = ceil_div(m, R);
    if (n_classes > FEW_CLASSES || tiles > FEW_TILES || (dense && !km_automatic_engine(km))) return TSVM_OK;
    if (tiles > 1) {
        if (!dense) TSVM_TRY(km_count_entries(km, st));
        if ((double) tiles * (dense ? (double) km->n * km->d_pad : (double) km->nnz) > 1.6e7) return TSVM_OK;
    }
    const int n_pairs = n_classes * (n_classes - 1) / 2;
    if (dense) {
        if (sizeof(float) * (size_t) R * km->d_pad + FewShared<8>::bytes(n_pairs) > 190 * 1024) return TSVM_OK;
    } else if (T_dev || tnnz <= 0 || tnnz > FEW_ENTRIES) return TSVM_OK;
    const size_t need = (size_t) FEW_TILES * 8 * n_pairs + FEW_TILES;
    if (km->few_cap < need) {
        pool_free(km->few_acc);
        km->few_acc = nullptr;
        km->few_cap = 0;
        TSVM_TRY(dev_alloc(&km->few_acc, need));
        TSVM_CUDA(cudaMemsetAsync(km->few_acc, 0, need * sizeof(double), st));
        km->few_cap = need;
    }
    FewArgs a;
    a.X = dense ? km->X : nullptr; a.ldx = km->ldx; a.val = km->val; a.row_ptr = km->row_ptr; a.col = km->col;
    a.n_sv = km->n; a.d = km->d; a.sd_sv = km->self_dot;
    a.T = T_dev; a.dt = dt; a.ldt = ldt; a.tval = tval_dev; a.trow_ptr = trow_ptr_dev; a.tcol = tcol_dev; a.m = m;
    a.fn = km->fn; a.coef = coef_dev; a.rho = rho_dev; a.n_classes = n_classes; a.n_pairs = n_pairs;
    a.start[0] = 0;
    for (int c = 0; c < n_classes; ++c) a.start[c + 1] = a.start[c] + sv_count_host[c];
    // the tickets lie at the end of the buffer, whatever the number of sums in front of them
    a.acc = km->few_acc; a.ticket = reinterpret_cast<int *>(km->few_acc + km->few_cap - FEW_TILES);
    a.dec = dec_dev; a.labels = labels_dev; a.overflow = km->status_host + 1;
    km->status_host[1] = 0;
    if (R == 1) TSVM_TRY(launch_few<1>(a, !dense, st));
    else if (R == 2) TSVM_TRY(launch_few<2>(a, !dense, st));
    else if (R == 4) TSVM_TRY(launch_few<4>(a, !dense, st));
    else TSVM_TRY(launch_few<8>(a, !dense, st));
    TSVM_CUDA(cudaStreamSynchronize(st));
    *taken = *(volatile int *) (km->status_host + 1) == 0;
    return TSVM_OK;
}

// All m rows, `batch` at a time, and a wait for the last of them.
static tsvm_status predict_slabs(tsvm_km *km_sv, const double *coef_dev, const std::vector<int> &start, const std::vector<int> &count,
                                 const double *rho_dev, int m, const float *T_dev, int dt, int ldt, const float *tval_dev,
                                 const int *trow_ptr_dev, const int *tcol_dev, double *dec_dev, int *labels_dev, bool fused,
                                 long long batch, long long ldk, cudaStream_t st) {
    const int n_sv = km_sv->n, n_classes = (int) start.size(), nb = n_classes * (n_classes - 1) / 2;
    float *K = nullptr;
    int *meta = nullptr, *sv_class = nullptr;
    double *dec_slab = nullptr;
    // test rows on the lanes: what that form needs of the support vectors, in place of their classes
    const int type = km_sv->fn.type;
    const bool rbf = type == TSVM_RBF || type == TSVM_PRECOMPUTED;
    const bool lanes = fused && m > LANES_ROWS && n_classes <= LANES_CLASSES && km_sv->plane_kind == 2 && (rbf || type == TSVM_LINEAR);
    float *columns = nullptr;
    const long long columns_ld = ((long long) n_sv + 255) / 256 * 256 + 256;       // (a block may read 255 past the last one)
    tsvm_status s = TSVM_OK;
    if (lanes) s = dev_alloc(&columns, (size_t) columns_ld * (3 + lanes_coefficients(n_classes)));
    else s = dev_alloc(&meta, (size_t) 2 * n_classes);
    if (s == TSVM_OK && !fused) s = dev_alloc(&K, (size_t) batch * ldk);
    if (s == TSVM_OK && fused && !lanes) s = dev_alloc(&sv_class, (size_t) n_sv);
    const bool by_pair = fused && sums_by_pair(n_classes);
    const long long slab_ld = (batch + 3) & ~3ll;
    if (s == TSVM_OK && (labels_dev || by_pair)) s = dev_alloc(&dec_slab, (size_t) slab_ld * nb);
    const bool by_argument = n_classes <= ARG_CLASSES;
    if (s == TSVM_OK && !by_argument) {
        cudaError_t e = cudaMemcpyAsync(meta, start.data(), sizeof(int) * n_classes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(meta + n_classes, count.data(), sizeof(int) * n_classes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);   // start/count are stack-local
        if (e != cudaSuccess) { set_error("predict: metadata copy failed: %s", cudaGetErrorString(e)); s = TSVM_ERR_CUDA; }
    }
    km_sv->status_host[0] = 0;
    auto run = [&]() -> tsvm_status {
        ClassCounts cc;
        for (int c = 0; c < n_classes && by_argument; ++c) cc.count[c] = count[c];
        if (lanes) {
            TSVM_LAUNCH(predict_columns_kernel, ceil_div(columns_ld, 256), 256, 0, st, cc, n_classes, n_sv, columns_ld,
                        lanes_coefficients(n_classes), coef_dev, km_sv->self_dot, km_sv->x_unscale, rbf, km_sv->fn.gamma, columns);
        } else if (by_argument) {
            TSVM_LAUNCH(class_tables_kernel, ceil_div(fused && n_sv > n_classes ? n_sv : n_classes, 256), 256, 0, st, cc,
                        n_classes, n_sv, meta, meta + n_classes, sv_class);
        } else if (fused) TSVM_LAUNCH(sv_class_kernel, ceil_div(n_sv, 256), 256, 0, st, sv_class, n_sv, meta, n_classes);
        for (long long r0 = 0; r0 < m; r0 += batch) {
            const int mm = (int) ((m - r0) < batch ? (m - r0) : batch);
            double *dec = labels_dev ? dec_slab : dec_dev + (size_t) r0 * nb;
            if (fused) {
                TSVM_TRY(fused_slab(km_sv, coef_dev, sv_class, columns, columns_ld, rho_dev, n_classes, r0, mm, T_dev, dt, ldt, tval_dev,
                                    trow_ptr_dev, tcol_dev, by_pair ? dec_slab : dec, by_pair ? slab_ld : 1, st));
                if (by_pair)
                    TSVM_LAUNCH(finish_slab_kernel, ceil_div(mm, 32), SLAB_THREADS, 0, st, dec_slab, slab_ld, mm, n_classes,
                                labels_dev ? nullptr : dec, labels_dev ? labels_dev + r0 : nullptr);
            } else {
                if (T_dev) TSVM_TRY(tsvm_km_rows_by_instances_dense(km_sv, T_dev + (size_t) r0 * ldt, mm, dt, ldt, K, ldk, st));
                else TSVM_TRY(tsvm_km_rows_by_instances_csr(km_sv, tval_dev, trow_ptr_dev + r0, tcol_dev, mm, 0, K, ldk, st));
                TSVM_LAUNCH(sum_kernel_values_kernel, mm, 256, 0, st, coef_dev, n_sv, meta, meta + n_classes, rho_dev, K,
                            ldk, dec, n_classes);
            }
            if (labels_dev && !by_pair)
                TSVM_TRY(launch_vote(dec, mm, n_classes, labels_dev + r0, st));
        }
        return TSVM_OK;
    };
    if (s == TSVM_OK) s = run();
    if (s == TSVM_OK) {
        const cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { set_error("predict failed: %s", cudaGetErrorString(e)); s = TSVM_ERR_CUDA; }
        else if (*(volatile int *) km_sv->status_host != 0) {       // written by the engine itself
            set_error("dense kernel-row engine reported status %d (a bounded wait ran out)", km_sv->status_host[0]);
            s = TSVM_ERR_DEVICE;
        }
    } else cudaStreamSynchronize(st);
    pool_free_many({K, meta, sv_class, dec_slab, columns}, s == TSVM_OK);      // (only this stream has used them)
    return s;
}

// labels_dev != nullptr: only the vote leaves the slab (sum_kernel_values_instant); dec_dev is then unused.
static tsvm_status predict_impl(tsvm_km *km_sv, const double *coef_dev, const int *sv_count_host, const double *rho_dev,
                                int n_classes, int m, const float *T_dev, int dt, int ldt, const float *tval_dev,
                                const int *trow_ptr_dev, const int *tcol_dev, long long tnnz, double *dec_dev,
                                int *labels_dev, size_t max_mem_bytes, cudaStream_t st) {
    const int n_sv = km_sv->n;
    int total = 0;
    std::vector<int> start(n_classes), count(n_classes);
    for (int c = 0; c < n_classes; ++c) { start[c] = total; count[c] = sv_count_host[c]; total += count[c]; }
    TSVM_REQUIRE(total == n_sv, "predict: support-vector counts sum to %d but the matrix holds %d", total, n_sv);
    km_sv->launched(st);
    bool taken = false;
    TSVM_TRY(predict_few(km_sv, coef_dev, sv_count_host, rho_dev, n_classes, m, T_dev, dt, ldt, tval_dev, trow_ptr_dev,
                         tcol_dev, tnnz, dec_dev, labels_dev, st, &taken));
    if (taken) { km_sv->waited(st); return TSVM_OK; }
    bool fused = false;
    TSVM_TRY(km_pair_engine_takes(km_sv, T_dev ? nullptr : tval_dev, T_dev ? nullptr : trow_ptr_dev, tcol_dev, m, st, &fused));
    const long long ldk = ((long long) n_sv + 3) & ~3ll;
    const bool scratch = labels_dev || sums_by_pair(n_classes);
    long long batch = fused ? fused_rows(km_sv, scratch ? (size_t) n_classes * (n_classes - 1) / 2 : 0) : 0;
    if (!fused) {
        // the kernel block of a slab must fit the budget (svmmodel.cpp:86-89 caps a batch at 10000 rows)
        size_t budget = max_mem_bytes;
        if (!budget) {
            // what all rows need, if that is no more than a sixteenth of the device
            budget = (size_t) (m < 10000 ? m : 10000) * (size_t) ldk * sizeof(float);
            const size_t most = device_memory_bytes() / 16;
            if (budget > most) budget = most;
        }
        batch = (long long) (budget / sizeof(float) / (size_t) ldk);
        if (batch > 10000) batch = 10000;
    }
    // slabs of equal size, in whole tiles
    if (fused && batch < m) batch = (ceil_div(m, ceil_div(m, batch)) + 255) / 256 * 256;
    if (batch > m) batch = m;
    if (batch < 1) batch = 1;
    // The size of the slab is a guess at what is free. Where the device has less (for the slab or for the staging scratch of
    // its rows), half of it will do: every slab writes all of its rows' results, so starting over is safe.
    tsvm_status s;
    for (;;) {
        s = predict_slabs(km_sv, coef_dev, start, count, rho_dev, m, T_dev, dt, ldt, tval_dev, trow_ptr_dev, tcol_dev, dec_dev,
                          labels_dev, fused, batch, ldk, st);
        if (s != TSVM_ERR_OOM || batch == 1) break;
        batch = (batch + 1) / 2;
    }
    if (s == TSVM_OK) km_sv->waited(st);
    return s;
}

extern "C" {

tsvm_status tsvm_predict_dec(tsvm_km *km_sv, const double *coef_dev, const int *sv_count_host, const double *rho_dev,
                             int n_classes, int m, const float *T_dev, int dt, int ldt, const float *tval_dev,
                             const int *trow_ptr_dev, const int *tcol_dev, long long tnnz, double *dec_dev,
                             size_t max_mem_bytes, void *stream) {
    TSVM_REQUIRE(km_sv && coef_dev && sv_count_host && rho_dev && dec_dev && n_classes >= 2 && m > 0,
                 "predict_dec: bad arguments");
    TSVM_REQUIRE(T_dev || trow_ptr_dev, "predict_dec: neither a dense nor a CSR test batch was given");
    return predict_impl(km_sv, coef_dev, sv_count_host, rho_dev, n_classes, m, T_dev, dt, ldt, tval_dev, trow_ptr_dev,
                        tcol_dev, tnnz, dec_dev, nullptr, max_mem_bytes, (cudaStream_t) stream);
}

tsvm_status tsvm_predict_labels(tsvm_km *km_sv, const double *coef_dev, const int *sv_count_host,
                                const double *rho_dev, int n_classes, int m, const float *T_dev, int dt, int ldt,
                                const float *tval_dev, const int *trow_ptr_dev, const int *tcol_dev, long long tnnz,
                                int *labels_dev, size_t max_mem_bytes, void *stream) {
    TSVM_REQUIRE(km_sv && coef_dev && sv_count_host && rho_dev && labels_dev && n_classes >= 2 && m > 0,
                 "predict_labels: bad arguments");
    TSVM_REQUIRE(T_dev || trow_ptr_dev, "predict_labels: neither a dense nor a CSR test batch was given");
    return predict_impl(km_sv, coef_dev, sv_count_host, rho_dev, n_classes, m, T_dev, dt, ldt, tval_dev, trow_ptr_dev,
                        tcol_dev, tnnz, nullptr, labels_dev, max_mem_bytes, (cudaStream_t) stream);
}

tsvm_status tsvm_vote(const double *dec_dev, int m, int n_classes, int *out_dev, void *stream) {
    TSVM_REQUIRE(dec_dev && out_dev && m > 0 && n_classes >= 2, "vote: bad arguments");
    return launch_vote(dec_dev, m, n_classes, out_dev, (cudaStream_t) stream);
}

}  // extern "C"
