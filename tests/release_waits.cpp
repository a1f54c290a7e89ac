// What the release of a SyncArray or DevicePtr waits for, on the stand-in runtime: its own stream if that is the only one it
// was used on and the one of the thread that releases it, else the device.
#include <thundersvm/syncarray.h>
#include <thundersvm/util/upload.h>
#include <cstdio>
#include <functional>
#include <memory>
#include <thread>

extern "C" {
void fake_reset_counts();
long long fake_device_waits();
long long fake_stream_waits();
}
using thundersvm::set_work_stream;

static void on(cudaStream_t s, const std::function<void()> &work) {
    std::thread([&] { set_work_stream(s); work(); set_work_stream(nullptr); }).join();
}
static int failed = 0;
static void expect(const char *what, bool device, const std::function<void()> &release) {
    fake_reset_counts();
    release();
    const bool waited = fake_device_waits() > 0;
    if (waited != device || (!device && fake_stream_waits() == 0)) { printf("%s: device waits %lld\n", what, fake_device_waits()); ++failed; }
}

int main() {
    cudaStream_t a, b;
    cudaStreamCreateWithFlags(&a, cudaStreamNonBlocking);
    cudaStreamCreateWithFlags(&b, cudaStreamNonBlocking);
    auto filled = [](cudaStream_t s) {
        std::unique_ptr<SyncArray<int>> p(new SyncArray<int>(1000));
        on(s, [&] { p->device_data(); });
        return p;
    };
    auto p = filled(a);
    expect("own stream", false, [&] { on(a, [&] { p.reset(); }); });
    p = filled(a);
    expect("another thread's stream", true, [&] { on(b, [&] { p.reset(); }); });
    p = filled(a);
    expect("a thread without a stream", true, [&] { p.reset(); });
    p = filled(nullptr);
    expect("default stream", true, [&] { p.reset(); });
    p = filled(a);
    on(b, [&] { p->device_data(); });
    expect("two streams", true, [&] { on(a, [&] { p.reset(); }); });
    p = filled(a);
    expect("resized by another thread", true, [&] { on(b, [&] { p->resize(10); }); });
    expect("after a resize", true, [&] { on(a, [&] { p->device_data(); }); on(b, [&] { p.reset(); }); });
    p = filled(a);
    auto q = filled(b);
    on(a, [&] { p->copy_from(*q); });
    expect("read by another array's copy", true, [&] { on(b, [&] { q.reset(); }); });
    expect("the copy", false, [&] { on(a, [&] { p.reset(); }); });
    thundersvm::DevicePtr<float> d;
    on(a, [&] { d = thundersvm::device_array<float>(100); });
    expect("device array, own stream", false, [&] { on(a, [&] { d.reset(); }); });
    on(a, [&] { d = thundersvm::device_array<float>(100); });
    expect("device array, another thread", true, [&] { on(b, [&] { d.reset(); }); });
    return failed;
}
