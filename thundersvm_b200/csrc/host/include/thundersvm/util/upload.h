// Host instances to device arrays. What bounds it is the host: a pageable copy of freshly zeroed memory ran at 2.5 GB/s
// (63 MB: 21 ms of page faults and zeros by one thread, 2 ms to fill it, 6.5 ms to copy). Here several threads write the
// device form straight into page-locked blocks that are kept between calls, and one block is on its way to the device
// while the next is filled: a fit of ten classes and 20,000 x 784 143 -> 54 ms.
#ifndef THUNDERSVM_UPLOAD_H
#define THUNDERSVM_UPLOAD_H
#include "../dataset.h"
#include <algorithm>
#include <cuda_runtime.h>
#include <memory>

namespace thundersvm {
struct DeviceFree {
    cudaStream_t used_on = nullptr;
    void operator()(void *p) const { device_free(p, used_on); }
};
template <typename T> using DevicePtr = std::unique_ptr<T, DeviceFree>;
// for the work stream of the thread that makes it; what else reads it waits by itself, as the handles do
template <typename T> DevicePtr<T> device_array(size_t count) {
    return DevicePtr<T>(static_cast<T *>(device_alloc(std::max<size_t>(count, 1) * sizeof(T))), DeviceFree{work_stream()});
}

// Two blocks of at least `bytes`, page-locked if the host has such memory, and what is needed to take turns with them
class UploadBlocks {
public:
    explicit UploadBlocks(size_t bytes, bool two);
    ~UploadBlocks();
    UploadBlocks(const UploadBlocks &) = delete;
    UploadBlocks &operator=(const UploadBlocks &) = delete;
    char *next();                                             // a block that no copy reads any more
    void send(void *dst, size_t bytes);                       // copies the block that next() gave out
    void finish();                                            // returns when everything has arrived
private:
    char *block_[2] = {nullptr, nullptr};
    cudaEvent_t sent_[2] = {nullptr, nullptr};
    bool busy_[2] = {false, false}, pinned_[2] = {false, false};
    int at_ = 1;
};

constexpr size_t UPLOAD_BLOCK = 4 << 20, UPLOAD_PARALLEL = 1 << 17;

// Row r becomes bytes [offset(r), offset(r + 1)) of dst: fill(r, p) writes them to p.
template <typename Offset, typename Fill>
void upload_rows(void *dst, size_t rows, Offset offset, Fill fill) {
    const size_t total = offset(rows);
    if (total == 0) return;
    size_t largest = 0;
    for (size_t r = 0; r < rows; ++r) largest = std::max(largest, offset(r + 1) - offset(r));
    const size_t room = std::min(total, std::max(size_t(UPLOAD_BLOCK), largest));
    UploadBlocks blocks(room, total > room);
    for (size_t r0 = 0; r0 < rows;) {
        size_t r1 = r0 + 1;
        while (r1 < rows && offset(r1 + 1) - offset(r0) <= room) ++r1;
        const size_t begin = offset(r0), bytes = offset(r1) - begin;
        char *p = blocks.next();
#pragma omp parallel for schedule(static) if (bytes > UPLOAD_PARALLEL)
        for (long r = (long) r0; r < (long) r1; ++r) fill((size_t) r, p + (offset((size_t) r) - begin));
        if (bytes) blocks.send(static_cast<char *>(dst) + begin, bytes);
        r0 = r1;
    }
    blocks.finish();
}

// Dense rows of ld floats, zero where a row has no such feature; row(k) gives the k-th one.
template <typename Row>
void upload_dense(float *dst, size_t rows, size_t ld, Row row) {
    upload_rows(dst, rows, [ld](size_t r) { return r * ld * sizeof(float); },
                [&](size_t r, char *p) {
                    float *x = reinterpret_cast<float *>(p);
                    std::memset(x, 0, ld * sizeof(float));
                    for (const DataSet::node &nd : row(r)) x[nd.index] = nd.value;
                });
}

// Entries and largest feature id of the instances
struct Extent { size_t nnz = 0; int max_index = 0; };
Extent extent_of(const DataSet::node2d &rows);

// Instances as CSR arrays on the device, ids as they are (1-based from LibSVM text).
class DeviceCsr {
public:
    explicit DeviceCsr(const DataSet::node2d &rows);
    const float *val() const { return val_.get(); }
    const int *col() const { return col_.get(); }
    const int *row_ptr() const { return row_ptr_.get(); }
    size_t nnz() const { return nnz_; }
private:
    DevicePtr<float> val_;
    DevicePtr<int> col_, row_ptr_;
    size_t nnz_ = 0;
};
}  // namespace thundersvm
#endif
