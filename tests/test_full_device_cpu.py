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


PREDICT = """
def predict(h, n_sv, m, classes=2, budget=0, dense=None, csr=None, labels=False):
    count = np.full(classes, n_sv // classes, np.int32)
    count[-1] += n_sv - count.sum()
    coef, rho = np.ones((classes - 1, n_sv)), np.zeros(classes * (classes - 1) // 2)
    out = np.zeros(m * max(1, len(rho)))
    batch = (p(dense), dense.shape[1], dense.shape[1], None, None, None) if csr is None else (None, 0, 0) + tuple(map(p, csr))
    nnz = 0 if csr is None else len(csr[0])
    f = L.tsvm_predict_labels if labels else L.tsvm_predict_dec
    return f(h, p(coef), p(count), p(rho), classes, m, *batch, C.c_longlong(nnz), p(out), C.c_size_t(budget), None)
"""


@pytest.mark.parametrize("free_mb", [300, 205, 64])
def test_prediction_takes_smaller_slabs(runtime, free_mb):
    """The stored kernel block of 10,000 x 20,000 (800 MB) does not fit; neither does the largest one that would leave no
    room for the staging panel (20 MB)."""
    fake_device.run_python(runtime, PREDICT + """
s, h, keep = csr(20000, 5000, 70)
check(s)
s, h2, rows = csr(10000, 5000, 70)
F.fake_set_free(%d * MB)
check(predict(h, 20000, 10000, csr=rows))
assert F.fake_largest_refused() >= 800000000
F.fake_set_free(0)
L.tsvm_release_cached_memory()
""" % free_mb)


def test_fused_prediction_takes_smaller_slabs(runtime):
    """4,096 staged rows of 4,096 features take 200 MB."""
    fake_device.run_python(runtime, PREDICT + """
s, h = dense(np.ones((2000, 4096), np.float32))
check(s)
F.fake_set_free(100 * MB)
check(predict(h, 2000, 5000, classes=3, dense=np.ones((5000, 4096), np.float32), labels=True))
""")


def test_prediction_without_room_for_one_row_is_refused(runtime):
    fake_device.run_python(runtime, PREDICT + """
s, h, keep = csr(20000, 5000, 70)
check(s)
s, h2, rows = csr(300, 5000, 70)
F.fake_set_free(0)
check(predict(h, 20000, 300, csr=rows), OOM)
F.fake_set_free(100 * MB)
check(predict(h, 20000, 300, csr=rows))
""")


@pytest.mark.parametrize("free_mb", [20, 35])
def test_sparse_data_without_room_for_a_dense_copy(runtime, free_mb):
    """30,000 x 200 as dense rows: 24 MB and two planes of 12 MB; the entries take 3.4 MB."""
    fake_device.run_python(runtime, """
F.fake_set_free(%d * MB)
s, h, keep = csr(30000, 200, 14)
check(s)
idx, out = np.arange(64, dtype=np.int32), np.zeros((64, 30000), np.float32)
check(L.tsvm_km_rows_by_index(h, p(idx), 64, p(out), C.c_longlong(30000), None))
""" % free_mb)


def test_a_solver_takes_the_room_of_a_dense_copy(runtime):
    """The smallest row buffer of a solve (184 MB) fits next to the entries, not next to the dense copy (48 MB) too. A
    solver that holds the handle keeps its storage as it is."""
    fake_device.run_python(runtime, """
s, h, keep = csr(30000, 200, 14)
check(s)
assert F.fake_used() > 48 * MB
F.fake_set_free(170 * MB)
s, S, keep2 = solver(h, 30000, 1024)
check(s)
L.tsvm_solver_destroy(S)
L.tsvm_km_destroy(h)
L.tsvm_release_cached_memory()
s, h, keep = csr(30000, 200, 14)
F.fake_set_free(250 * MB)
s, S, keep2 = solver(h, 30000, 1024)
check(s)
F.fake_set_free(170 * MB)
s, S2, keep3 = solver(h, 30000, 1024)
check(s, OOM)
L.tsvm_solver_destroy(S)
L.tsvm_km_destroy(h)
""")


def test_dense_data_without_room_for_planes(runtime):
    """The planes are for the engines that read them: without room the handle is made, and a CUDA-core row can be asked for."""
    fake_device.run_python(runtime, """
X = np.ones((30000, 200), np.float32)
F.fake_set_free(28 * MB)
s, h = dense(X)
check(s)
idx, out = np.arange(64, dtype=np.int32), np.zeros((64, 30000), np.float32)
rows = lambda: L.tsvm_km_rows_by_index(h, p(idx), 64, p(out), C.c_longlong(30000), None)
check(rows(), OOM)
check(L.tsvm_km_set_dense_engine(h, 1))
check(rows())
F.fake_set_free(100 * MB)
check(L.tsvm_km_set_dense_engine(h, 0))
check(rows())
""")


def test_row_cache_leaves_room_for_the_rest(runtime):
    """A quarter of the rows wanted (384 MB) fits to within 2 MB, and the working set's block alone takes 4 MB."""
    fake_device.run_python(runtime, """
s, h = dense(np.ones((20000, 64), np.float32))
check(s)
F.fake_set_free(386 * MB)
s, S, keep = solver(h, 20000)
check(s)
idx, out = np.arange(512, dtype=np.int32), np.zeros((512, 20000), np.float32)
check(L.tsvm_km_rows_by_index(h, p(idx), 512, p(out), C.c_longlong(20000), None))
""")


HOST_MODEL = """
import host_api
H = host_api.load()
rng = np.random.default_rng(0)
def model(n_sv, d, per_row):
    rows = [" ".join("%d:1" % c for c in np.sort(rng.choice(d, per_row, replace=False)) + 1) for _ in range(n_sv)]
    head = ["svm_type c_svc", "kernel_type rbf", "gamma 0.5", "nr_class 2", "total_sv %d" % n_sv, "rho 0.1", "label 0 1",
            "nr_sv %d %d" % (n_sv // 2, n_sv - n_sv // 2), "SV"]
    m = H.model_new(0)
    H.load_from_string_scikit(m, "\\n".join(head + ["1 " + r for r in rows] + [""]).encode())
    assert H.n_sv(m) == n_sv
    return m
def label(m, n_rows, d, per_row):
    rp = np.arange(0, n_rows * per_row + 1, per_row, dtype=np.int32)
    col = np.tile(np.arange(1, per_row + 1, dtype=np.int32), n_rows)
    val, out = np.ones(len(col), np.float32), np.zeros(n_rows, np.float32)
    return H.sparse_predict(n_rows, host_api.p(val, host_api.f32p), host_api.p(rp, host_api.i32p),
                            host_api.p(col, host_api.i32p), m, host_api.p(out, host_api.f32p), 0)
"""


def test_host_prediction_keeps_to_the_entries(runtime):
    """4,000 support vectors of 2,000 features, 2 % set: 32 MB as dense rows and as much for the planes, 1.3 MB as entries."""
    fake_device.run_python(runtime, HOST_MODEL + """
m = model(4000, 2000, 42)
for free in (20, 45, 200):
    F.fake_set_free(free * MB)
    assert label(m, 100, 2000, 42) == 0
    L.tsvm_release_cached_memory()
""")


def test_uploads_without_page_locked_memory(runtime):
    """The host may refuse page-locked memory (a limit, a full machine): the instances go through ordinary memory then."""
    fake_device.run_python(runtime, HOST_MODEL + """
m = model(400, 2000, 42)
assert label(m, 100, 2000, 42) == 0
L.tsvm_release_cached_memory()
F.fake_refuse_pinned(1)
assert label(m, 100, 2000, 42) == 0
assert label(m, 40000, 2000, 42) == 0           # more than one block
""")
