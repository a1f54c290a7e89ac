// Host runtime pieces shared by the model layer: verbosity switch, device-memory helpers behind
// SyncArray, the parameter name tables and the two metrics.
#include <thundersvm/thundersvm.h>
#include <thundersvm/syncarray.h>
#include <thundersvm/svmparam.h>
#include <thundersvm/util/metric.h>
#include <thundersvm/util/upload.h>
#include <cuda_runtime.h>
#include "../common.cuh"

namespace thundersvm {
bool g_verbose = true;
void set_verbose(bool on) { g_verbose = on; }

static void cuda_ok(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return;
    cudaGetLastError();                                               // reported here, not by the next launch too
    if (e == cudaErrorMemoryAllocation) throw std::bad_alloc();       // reference: util/common.h:33-39
    LOG(FATAL) << what << ": " << cudaGetErrorString(e);
}
// SyncArray memory comes from the library's pool (a model trains one binary problem per class pair, each
// with its own arrays)
void *device_alloc(size_t bytes) {
    void *p = nullptr;
    const tsvm_status s = tsvm::pool_alloc(&p, bytes ? bytes : 1);
    if (s == TSVM_ERR_OOM) throw std::bad_alloc();                    // reference: util/common.h:33-39
    if (s != TSVM_OK) LOG(FATAL) << "device allocation: " << tsvm_last_error();
    return p;
}
static thread_local cudaStream_t tl_stream = nullptr;
cudaStream_t work_stream() { return tl_stream; }
void set_work_stream(cudaStream_t s) { tl_stream = s; }
// Copies are ordered on the calling thread's stream; those that touch host memory return when they are done,
// as cudaMemcpy does.
void copy_to_device(void *dst, const void *src, size_t bytes) {
    cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, tl_stream), "H2D copy");
    cuda_ok(cudaStreamSynchronize(tl_stream), "H2D copy");
}
void copy_to_host(void *dst, const void *src, size_t bytes) {
    cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, tl_stream), "D2H copy");
    cuda_ok(cudaStreamSynchronize(tl_stream), "D2H copy");
}
void copy_on_device(void *dst, const void *src, size_t bytes) {
    cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, tl_stream), "D2D copy");
}
void device_free(void *p, cudaStream_t used_on) {
    if (!p) return;
    const bool own = used_on && used_on == tl_stream;
    if (own) cudaStreamSynchronize(tl_stream);
    tsvm::pool_free_many({p}, own);
}
// The driver is asked for the free memory only where it matters (a driver lock, at times tens of milliseconds): what fits
// a hundredth of the device is tried first, and a device that full fails the allocation (with_room tries again).
static thread_local int tl_room_asked = 0;
RoomAsked::RoomAsked() { ++tl_room_asked; }
RoomAsked::~RoomAsked() { --tl_room_asked; }
bool device_has_room(double bytes) {
    if (!tl_room_asked && bytes < 0.01 * (double) tsvm::device_memory_bytes()) return true;
    size_t free_b = 0, total_b = 0;
    return cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && bytes < 0.6 * (double) free_b;
}
void device_zero(void *p, size_t bytes) { cuda_ok(cudaMemsetAsync(p, 0, bytes, tl_stream), "cudaMemset"); }

UploadBlocks::UploadBlocks(size_t bytes, bool two) {
    for (int b = 0; b < (two ? 2 : 1); ++b) {
        pinned_[b] = tsvm::pinned_alloc(reinterpret_cast<void **>(block_ + b), bytes) == TSVM_OK;
        if (!pinned_[b]) {                        // the host has none to give: copies through the driver's own, slower
            block_[b] = static_cast<char *>(std::malloc(bytes));
            if (!block_[b]) throw std::bad_alloc();
        }
        if (two) cuda_ok(cudaEventCreateWithFlags(sent_ + b, cudaEventDisableTiming), "event");
    }
}
UploadBlocks::~UploadBlocks() {
    if (busy_[0] || busy_[1]) cudaStreamSynchronize(tl_stream);
    for (int b = 0; b < 2; ++b) {
        if (sent_[b]) cudaEventDestroy(sent_[b]);
        if (block_[b]) { if (pinned_[b]) tsvm::pinned_free(block_[b]); else std::free(block_[b]); }
    }
}
char *UploadBlocks::next() {
    at_ = block_[1] ? 1 - at_ : 0;
    if (busy_[at_]) cuda_ok(sent_[at_] ? cudaEventSynchronize(sent_[at_]) : cudaStreamSynchronize(tl_stream), "H2D copy");
    busy_[at_] = false;
    return block_[at_];
}
void UploadBlocks::send(void *dst, size_t bytes) {
    cuda_ok(cudaMemcpyAsync(dst, block_[at_], bytes, cudaMemcpyHostToDevice, tl_stream), "H2D copy");
    if (sent_[at_]) cuda_ok(cudaEventRecord(sent_[at_], tl_stream), "event");
    busy_[at_] = true;
}
void UploadBlocks::finish() {
    cuda_ok(cudaStreamSynchronize(tl_stream), "H2D copy");
    busy_[0] = busy_[1] = false;
}

Extent extent_of(const DataSet::node2d &rows) {
    size_t nnz = 0;
    int mx = 0;
#pragma omp parallel for schedule(static) reduction(+ : nnz) reduction(max : mx) if (rows.size() > 1024)
    for (long r = 0; r < (long) rows.size(); ++r) {
        nnz += rows[r].size();
        for (auto &nd : rows[r]) if (nd.index > mx) mx = nd.index;
    }
    Extent e;
    e.nnz = nnz; e.max_index = mx;
    return e;
}

DeviceCsr::DeviceCsr(const DataSet::node2d &rows) {
    const size_t m = rows.size();
    vector<int> rp(m + 1, 0);
    for (size_t r = 0; r < m; ++r) rp[r + 1] = rp[r] + (int) rows[r].size();
    nnz_ = rp[m];
    auto offset = [&](size_t r) { return (size_t) rp[r] * 4; };
    row_ptr_ = device_array<int>(m + 1);
    val_ = device_array<float>(nnz_);
    col_ = device_array<int>(nnz_);
    copy_to_device(row_ptr_.get(), rp.data(), (m + 1) * sizeof(int));
    upload_rows(val_.get(), m, offset, [&](size_t r, char *p) {
        float *v = reinterpret_cast<float *>(p);
        for (auto &nd : rows[r]) *v++ = nd.value;
    });
    upload_rows(col_.get(), m, offset, [&](size_t r, char *p) {
        int *c = reinterpret_cast<int *>(p);
        for (auto &nd : rows[r]) *c++ = nd.index;
    });
}

std::atomic<size_t> &total_memory_size() {
    static std::atomic<size_t> bytes{0};
    return bytes;
}
}  // namespace thundersvm

const char *SvmParam::kernel_type_name[6] = {"linear", "polynomial", "rbf", "sigmoid", "precomputed", "NULL"};
const char *SvmParam::svm_type_name[6] = {"c_svc", "nu_svc", "one_class", "epsilon_svr", "nu_svr", "NULL"};

string Accuracy::name() { return "Accuracy"; }
float_type Accuracy::score(const vector<float_type> &predict_y, const vector<float_type> &ground_truth_y) {
    size_t hits = 0;
    for (size_t i = 0; i < predict_y.size(); ++i) hits += predict_y[i] == ground_truth_y[i];
    return hits / (float) ground_truth_y.size();
}
string MSE::name() { return "Mean Squared Error"; }
float_type MSE::score(const vector<float_type> &predict_y, const vector<float_type> &ground_truth_y) {
    float_type acc = 0;
    for (size_t i = 0; i < predict_y.size(); ++i) {
        const float_type e = predict_y[i] - ground_truth_y[i];
        acc += e * e;
    }
    return acc / predict_y.size();
}
