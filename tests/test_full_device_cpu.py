"""What the host code does when the device is (nearly) full, on the stand-in runtime of fake_device.py."""
import fake_device
import pytest


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    from thundersvm_b200 import build
    build.build()
    return fake_device.compile_runtime(tmp_path_factory.mktemp("fake"))


def test_a_refused_allocation_is_reported_once(runtime):
    """The call that ran out of memory says so; the next one, with room, does not inherit the runtime's last error."""
    fake_device.run_python(runtime, """
X = np.ones((4000, 64), np.float32)
F.fake_set_free(MB // 2)
s, h = dense(X)
check(s, OOM)
F.fake_set_free(1024 * MB)
s, h = dense(X)
check(s)
""")


def test_row_cache_takes_what_is_there(runtime):
    """20,000 instances: 1.6 GB of rows wanted, 400 MB free, 123 MB are enough."""
    fake_device.run_python(runtime, """
s, h = dense(np.ones((20000, 64), np.float32))
check(s)
F.fake_set_free(400 * MB)
s, S, keep = solver(h, 20000)
check(s)
assert F.fake_largest_refused() > 1400 * MB, F.fake_largest_refused()
""")
