// KernelMatrix, CSMOSolver and NuSMOSolver: thin forwards to the C ABI (include/thundersvm_b200.h).
// Reference behaviour: src/thundersvm/kernelmatrix.cpp:183-316, src/thundersvm/solver/csmosolver.cpp:10-121.
#include <thundersvm/kernelmatrix.h>
#include <thundersvm/solver/csmosolver.h>
#include <thundersvm/solver/nusmosolver.h>
#include <cuda_runtime.h>
#include <mutex>
#include "../common.cuh"

namespace {
void b200_check(tsvm_status s) {
    if (s == TSVM_OK) return;
    if (s == TSVM_ERR_OOM) throw std::bad_alloc();
    LOG(FATAL) << "thundersvm_b200: " << tsvm_last_error();
}
}  // namespace

KernelMatrix::KernelMatrix(const DataSet::node2d &instances, SvmParam param) : param_(param) {
    n_instances_ = instances.size();
    CHECK(n_instances_ > 0) << "KernelMatrix needs at least one instance";
    const thundersvm::Extent ext = thundersvm::extent_of(instances);
    n_features_ = (size_t) ext.max_index + 1;   // column 0 stays empty for one-based data (kernelmatrix.cpp:200-206)
    nnz_ = ext.nnz;
    // Storage: the tensor-core engine wants a dense row-major matrix; it pays off unless the data
    // is very sparse (then the CSR engine touches far fewer bytes) or the three dense planes would
    // not fit next to the kernel-row buffer.
    const double density = (double) nnz_ / ((double) n_instances_ * n_features_);
    const double dense_bytes = 3.0 * n_instances_ * ((n_features_ + 3) & ~3ul) * 4.0 + 1024.0 * n_instances_ * 4.0;
    dense_ = (density >= 0.02 || n_features_ <= 256) && thundersvm::device_has_room(dense_bytes);
    if (dense_) {
        const size_t ld = (n_features_ + 3) & ~(size_t) 3;
        own_x_ = thundersvm::device_array<float>(n_instances_ * ld);
        thundersvm::upload_dense(own_x_.get(), n_instances_, ld,
                                 [&](size_t r) -> const vector<DataSet::node> & { return instances[r]; });
        b200_check(tsvm::km_create_dense(own_x_.get(), (int) n_instances_, (int) n_features_, (int) ld, TSVM_DEVICE, true,
                                         param.kernel_type, param.degree, (float) param.gamma, (float) param.coef0,
                                         thundersvm::work_stream(), &km_));
    } else {
        own_csr_.reset(new thundersvm::DeviceCsr(instances));
        b200_check(tsvm_km_create_csr(own_csr_->val(), own_csr_->row_ptr(), own_csr_->col(), (int) n_instances_,
                                      (int) n_features_, TSVM_DEVICE, param.kernel_type, param.degree,
                                      (float) param.gamma, (float) param.coef0, thundersvm::work_stream(), &km_));
        km_->nnz = (long long) nnz_;
    }
    thundersvm::total_memory_size() += (dense_ ? (size_t) dense_bytes : nnz_ * 8 + n_instances_ * 12);
}

KernelMatrix::KernelMatrix(const float *X_dev, size_t d, size_t ld, size_t r0, size_t n0, size_t r1, size_t n1,
                           SvmParam param) : param_(param) {
    n_instances_ = n0 + n1;
    n_features_ = d;
    nnz_ = n_instances_ * d;
    dense_ = true;
    CHECK(n_instances_ > 0) << "KernelMatrix needs at least one instance";
    own_x_ = thundersvm::device_array<float>(n_instances_ * ld);
    thundersvm::copy_on_device(own_x_.get(), X_dev + r0 * ld, n0 * ld * sizeof(float));
    thundersvm::copy_on_device(own_x_.get() + n0 * ld, X_dev + r1 * ld, n1 * ld * sizeof(float));
    b200_check(tsvm::km_create_dense(own_x_.get(), (int) n_instances_, (int) d, (int) ld, TSVM_DEVICE, true, param.kernel_type,
                                     param.degree, (float) param.gamma, (float) param.coef0, thundersvm::work_stream(), &km_));
    const double dense_bytes = 3.0 * n_instances_ * ((n_features_ + 3) & ~3ul) * 4.0 + 1024.0 * n_instances_ * 4.0;
    thundersvm::total_memory_size() += (size_t) dense_bytes;
}

KernelMatrix::~KernelMatrix() {
    if (km_) {
        const double dense_bytes = 3.0 * n_instances_ * ((n_features_ + 3) & ~3ul) * 4.0 + 1024.0 * n_instances_ * 4.0;
        thundersvm::total_memory_size() -= (dense_ ? (size_t) dense_bytes : nnz_ * 8 + n_instances_ * 12);
        tsvm_km_destroy(km_);
    }
}

void KernelMatrix::get_rows(const SyncArray<int> &idx, SyncArray<kernel_type> &kernel_rows) const {
    CHECK_GE(kernel_rows.size(), idx.size() * n_instances_) << "kernel_rows memory is too small";
    b200_check(tsvm_km_rows_by_index(km_, idx.device_data(), (int) idx.size(), kernel_rows.device_data(),
                                     (long long) n_instances_, thundersvm::work_stream()));
}

void KernelMatrix::get_rows(const DataSet::node2d &instances, SyncArray<kernel_type> &kernel_rows) const {
    CHECK_GE(kernel_rows.size(), instances.size() * n_instances_) << "kernel_rows memory is too small";
    if (instances.empty()) return;
    const thundersvm::DeviceCsr c(instances);
    b200_check(tsvm_km_rows_by_instances_csr(km_, c.val(), c.row_ptr(), c.col(), (int) instances.size(),
                                             (long long) c.nnz(), kernel_rows.device_data(),
                                             (long long) n_instances_, thundersvm::work_stream()));
    cudaStreamSynchronize(thundersvm::work_stream());
}

// (copied when someone asks: a solve does not, and the copy is a wait)
const SyncArray<kernel_type> &KernelMatrix::diag() const {
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (diag_.size() != n_instances_) {
        diag_.resize(n_instances_);
        thundersvm::copy_to_host(diag_.host_data(), km_->diag, sizeof(kernel_type) * n_instances_);
    }
    return diag_;
}

int CSMOSolver::solver_kind() const { return TSVM_SOLVER_C; }
int NuSMOSolver::solver_kind() const { return for_svr ? TSVM_SOLVER_NU_SVR : TSVM_SOLVER_NU_SVC; }

void CSMOSolver::solve(const KernelMatrix &k_mat, const SyncArray<int> &y, SyncArray<float_type> &alpha,
                       float_type &rho, SyncArray<float_type> &f_val, float_type eps, float_type Cp, float_type Cn,
                       int ws_size, int max_iter) const {
    LOG(INFO) << "training start";
    tsvm_solve_stats st;
    double rho_out = 0;
    b200_check(tsvm_smo_solve(k_mat.handle(), solver_kind(), y.device_data(), alpha.device_data(), f_val.device_data(),
                              eps, Cp, Cn, ws_size, max_iter, &rho_out, &st, thundersvm::work_stream()));
    rho = rho_out;
    LOG(INFO) << "global iter = " << st.outer_iters - 1 << ", total local iter = " << st.local_iters << ", diff = "
              << st.final_diff;
    LOG(INFO) << "training finished";
    LOG(INFO) << "obj = " << st.objective;
}
