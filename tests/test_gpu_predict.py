"""Prediction on the GPU against the oracle and the committed reference outputs.
Tolerance: decision values 1e-3 absolute, labels >= 99.9 % agreement."""
import os

import numpy as np
import pytest

from oracle import port_binding as P

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_multiclass_decision_values_and_vote(capi):
    import torch
    rng = np.random.default_rng(3)
    nc, d, n_sv, m = 4, 24, 230, 157
    SVd = rng.standard_normal((n_sv, d)).astype(np.float32)
    T = rng.standard_normal((m, d)).astype(np.float32)
    cnt = np.array([60, 50, 70, 50], dtype=np.int32)
    coef = rng.standard_normal((nc - 1, n_sv))
    rho = rng.standard_normal(nc * (nc - 1) // 2)
    want = P.predict_dec(P.Csr(dense=SVd), coef.reshape(-1), cnt, rho, nc, P.Csr(dense=T), gamma=0.05)
    for dense_sv in (True, False):
        if dense_sv:
            km = capi.KernelMatrix(dense=_t(SVd), gamma=0.05)
        else:
            c = P.Csr(dense=SVd)
            km = capi.KernelMatrix(csr=(_t(c.val), _t(c.row_ptr), _t(c.col)), d=d, gamma=0.05)
        for budget in (0, 64 * 1024):            # one batch / many small batches
            dec = capi.predict_dec(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, dense=_t(T), max_mem_bytes=budget)
            assert np.max(np.abs(dec.cpu().numpy() - want)) < 1e-3
            got = capi.vote(dec, nc).cpu().numpy()
            assert np.mean(got == P.vote(want, nc)) >= 0.999


def test_reference_fixture_decision_values(capi, golden_dir):
    """Support vectors / coefficients / rho of the reference-trained models (tests/golden) -> the
    reference's own decision values on its fixture data set."""
    g = np.load(os.path.join(golden_dir, "test_dataset.npz"))
    val, rp, col, d, y = g["val"], g["row_ptr"], g["col"], int(g["d"]), g["y"]
    n = len(rp) - 1
    Xd = np.zeros((n, d), np.float32)
    Xd[np.repeat(np.arange(n), np.diff(rp)), col] = val
    for tag, nc in (("svc", 3), ("svr", 2), ("oneclass", 2), ("nusvr", 2)):
        sv = Xd[g[tag + "_sv_ind"]]
        km = capi.KernelMatrix(dense=_t(sv), gamma=0.5)
        cnt = g[tag + "_n_sv"]
        dec = capi.predict_dec(km, _t(g[tag + "_coef"]), cnt, _t(g[tag + "_rho"]), nc, dense=_t(Xd)).cpu().numpy()
        assert np.max(np.abs(dec - g[tag + "_dec"])) < 1e-3
    # labels of the 3-class model: accuracy 0.98 (src/test/test_svc.cpp:33-37)
    sv = Xd[g["svc_sv_ind"]]
    km = capi.KernelMatrix(dense=_t(sv), gamma=0.5)
    dec = capi.predict_dec(km, _t(g["svc_coef"]), g["svc_n_sv"], _t(g["svc_rho"]), 3, dense=_t(Xd))
    labels = np.array([0.0, 2.0, 3.0])[capi.vote(dec, 3).cpu().numpy()]
    assert np.array_equal(labels, g["svc_pred"])
    assert abs((labels == y).mean() - 0.98) < 1e-5


def _fused_case(capi, nc, cnt, d, m, kernel="rbf", gamma=0.02, coef0=0.0, degree=3, engine=None, csr_batch=False,
                seed=5):
    """Dense support vectors with more than 32 features: the coefficient sums are the contraction's epilogue."""
    rng = np.random.default_rng(seed)
    cnt = np.asarray(cnt, dtype=np.int32)
    n_sv = int(cnt.sum())
    SVd = (rng.standard_normal((n_sv, d)) * (rng.random((n_sv, d)) < 0.6)).astype(np.float32)
    T = (rng.standard_normal((m, d)) * (rng.random((m, d)) < 0.6)).astype(np.float32)
    coef = rng.standard_normal((nc - 1, n_sv)) * 3
    rho = rng.standard_normal(nc * (nc - 1) // 2)
    kw = dict(kernel=kernel, gamma=gamma, coef0=coef0, degree=degree)
    want = P.predict_dec(P.Csr(dense=SVd), coef.reshape(-1), cnt, rho, nc, P.Csr(dense=T), **kw)
    km = capi.KernelMatrix(dense=_t(SVd), **kw)
    if engine:
        km.set_dense_engine(engine)
    if csr_batch:
        c = P.Csr(dense=T)
        nz = c.val != 0                          # drop the explicit zeros: a genuinely sparse batch
        rp = np.concatenate([[0], np.cumsum(np.add.reduceat(nz, c.row_ptr[:-1]))]).astype(np.int32)
        batch = dict(csr=(_t(c.val[nz]), _t(rp), _t(c.col[nz])))
    else:
        batch = dict(dense=_t(T))
    dec = capi.predict_dec(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, **batch).cpu().numpy()
    scale = max(1.0, float(np.max(np.abs(want))))
    assert np.max(np.abs(dec - want)) < 1e-3 * scale, np.max(np.abs(dec - want))
    lab = capi.predict_labels(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, **batch).cpu().numpy()
    assert np.array_equal(lab, capi.vote(_t(dec), nc).cpu().numpy())
    assert np.mean(lab == P.vote(want, nc)) >= 0.999
    km.close()


@pytest.mark.parametrize("engine", [None, "tensor2"])
def test_fused_prediction_multiclass_ragged_classes(capi, engine):
    """Class blocks that start and end inside a 128-instance tile, a tail tile, a tail row block."""
    _fused_case(capi, 4, [300, 37, 401, 262], d=200, m=700, engine=engine)


def test_fused_prediction_binary_tails_and_sparse_batch(capi):
    _fused_case(capi, 2, [513, 258], d=136, m=257)
    _fused_case(capi, 2, [100, 29], d=72, m=5, csr_batch=True)
    _fused_case(capi, 3, [1, 1, 1], d=40, m=300)


@pytest.mark.parametrize("kernel,kw", [("linear", {}), ("poly", dict(gamma=0.01, coef0=0.5, degree=3)),
                                       ("sigmoid", dict(gamma=0.01, coef0=0.1))])
def test_fused_prediction_other_kernels(capi, kernel, kw):
    _fused_case(capi, 3, [150, 200, 90], d=96, m=333, kernel=kernel, **kw)


@pytest.mark.parametrize("nc", [3, 4, 5, 10, 11, 32, 33])
def test_fused_prediction_numbers_of_classes(capi, nc):
    """Around the numbers of coefficients and classes where the fused path changes: 3 and 4 coefficients, 9 and 10, 32 and 33
    classes; rows that are no multiple of 32, classes of one and of 33 support vectors."""
    _fused_case(capi, nc, [1 + 32 * (c % 2) for c in range(nc)], d=40, m=97)


@pytest.mark.parametrize("d,gamma", [(64, 0.02), (2050, 5e-4)])
def test_fused_prediction_many_classes(capi, d, gamma):
    """20 classes: 19 coefficient rows per support vector (more than the shared-memory table holds) and 190 pairs; with 2,050
    features in two launches over the test rows."""
    _fused_case(capi, 20, [17 + 3 * c for c in range(20)], d=d, m=4500, gamma=gamma)


@pytest.mark.parametrize("m", [192, 193, 256, 257, 700])
@pytest.mark.parametrize("kernel", ["rbf", "linear"])
@pytest.mark.parametrize("cnt", [[1, 0], [16, 15], [130, 127], [20, 12, 31], [256, 1, 0, 255], [9, 16, 17, 0, 1, 64, 33, 2, 5, 100],
                                 [40] * 11])
def test_fused_prediction_rows_on_the_lanes(capi, m, kernel, cnt):
    """From 193 rows on the test rows lie on the lanes and the support vectors on the columns: row tiles and their remainders,
    blocks of columns and their remainders, classes that begin and end at a group of 16 columns, inside one, several in one,
    none in a class; the last number of classes of that form and the first beyond it. Against sums in FP64: kernel values
    and products are FP32, the error of a sum of n products stays below (n + 20) 2^-24 times the sum of their magnitudes."""
    rng = np.random.default_rng(m + len(cnt))
    cnt = np.asarray(cnt, dtype=np.int32)
    nc, n_sv, d, gamma = len(cnt), int(cnt.sum()), 65, 0.02
    SV, T = (rng.standard_normal((k, d)).astype(np.float32) for k in (n_sv, m))
    coef, rho = rng.standard_normal((nc - 1, n_sv)), rng.standard_normal(nc * (nc - 1) // 2)
    dots = T.astype(np.float64) @ SV.T.astype(np.float64)
    K = dots
    if kernel == "rbf":
        K = np.exp(-gamma * ((T.astype(np.float64) ** 2).sum(1)[:, None] + (SV.astype(np.float64) ** 2).sum(1)[None] - 2 * dots))
    own = np.repeat(np.arange(nc), cnt)
    want, size = [], []
    for i in range(nc):
        for j in range(i + 1, nc):
            c = np.where(own == i, coef[j - 1], 0.0) + np.where(own == j, coef[i], 0.0)
            want.append(K @ c - rho[len(want)])
            size.append(np.abs(K) @ np.abs(c))
    want, size = np.stack(want, 1), np.stack(size, 1)
    # values: up to 2 gamma |x| |y| log2 e 2^-24 relative in the exponent (RBF), the dot's own 2^-24 sum of magnitudes (linear)
    term = np.abs(T).astype(np.float64) @ np.abs(SV).T.astype(np.float64)
    loose = (K * gamma * 4 * (term + (T ** 2).sum(1)[:, None] + (SV ** 2).sum(1)[None]) if kernel == "rbf" else 4 * term) * np.abs(coef).sum(0)
    km = capi.KernelMatrix(dense=_t(SV), kernel=kernel, gamma=gamma)
    dec = capi.predict_dec(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, dense=_t(T))
    bound = 2.0 ** -24 * ((n_sv + 20) * size + loose.sum(1)[:, None]) + 1e-12
    assert np.all(np.abs(dec.cpu().numpy() - want) <= bound), np.max(np.abs(dec.cpu().numpy() - want) / bound)
    lab = capi.predict_labels(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, dense=_t(T))
    assert np.array_equal(lab.cpu().numpy(), capi.vote(dec, nc).cpu().numpy())
    km.close()


def _sums_in_fp64(SV, T, kernel, gamma, cnt, coef, rho):
    """Decision values in FP64, and the bound on the error of FP32 kernel values and products: (n + 20) 2^-24 times the sum of
    the magnitudes of a pair's n products, and the values' own errors - the exponent's 2 gamma |x| |y| 2^-24 and more (RBF), the
    dot's 2^-24 times its sum of magnitudes (linear)."""
    A, B = T.astype(np.float64), SV.astype(np.float64)
    dots, squares = A @ B.T, (A ** 2).sum(1)[:, None] + (B ** 2).sum(1)[None]
    K = np.exp(-gamma * (squares - 2 * dots)) if kernel == "rbf" else dots
    term = np.abs(A) @ np.abs(B).T
    loose = (K * gamma * 4 * (term + squares) if kernel == "rbf" else 4 * term) @ np.abs(coef).sum(0)
    own, want, size = np.repeat(np.arange(len(cnt)), cnt), [], []
    for i in range(len(cnt)):
        for j in range(i + 1, len(cnt)):
            c = np.where(own == i, coef[j - 1], 0.0) + np.where(own == j, coef[i], 0.0)
            want.append(K @ c - rho[len(want)])
            size.append(np.abs(K) @ np.abs(c))
    return np.stack(want, 1), 2.0 ** -24 * ((len(own) + 20) * np.stack(size, 1) + loose[:, None]) + 1e-12


def _sums_case(capi, km, SV, T, kernel, gamma, cnt, seed, batch):
    rng = np.random.default_rng(seed)
    nc, n_sv = len(cnt), int(np.sum(cnt))
    coef, rho = rng.standard_normal((nc - 1, n_sv)), rng.standard_normal(nc * (nc - 1) // 2)
    want, bound = _sums_in_fp64(SV, T, kernel, gamma, cnt, coef, rho)
    dec = capi.predict_dec(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, **batch)
    assert np.all(np.abs(dec.cpu().numpy() - want) <= bound), np.max(np.abs(dec.cpu().numpy() - want) / bound)
    lab = capi.predict_labels(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, **batch).cpu().numpy()
    # labels are the vote over a second call's sums, whose order may differ: rows without a value in doubt
    sure = (np.abs(want) > bound).all(1)
    assert sure.any() and np.array_equal(lab[sure], capi.vote(dec, nc).cpu().numpy()[sure])
    km.close()


@pytest.mark.parametrize("d", [127, 128, 129, 256, 257, 300, 784])
@pytest.mark.parametrize("m", [193, 513])
@pytest.mark.parametrize("kernel", ["rbf", "linear"])
@pytest.mark.parametrize("cnt", [[130, 127], [20, 12, 31], [300, 1, 0, 255], [57] * 10, [9, 16, 17, 0, 1, 64, 33, 2, 5, 300]])
def test_fused_prediction_rows_on_the_lanes_numbers_of_features(capi, d, m, kernel, cnt):
    """Test rows on the lanes with one promotion unit (up to 128 features), where the sums are taken from tensor memory, and with
    several, where they stay in registers: one, three and nine coefficients, more than one block of support vectors."""
    rng = np.random.default_rng(d + m)
    SV, T = (rng.standard_normal((k, d)).astype(np.float32) for k in (sum(cnt), m))
    km = capi.KernelMatrix(dense=_t(SV), kernel=kernel, gamma=1.0 / d)
    _sums_case(capi, km, SV, T, kernel, 1.0 / d, cnt, len(cnt), dict(dense=_t(T)))


@pytest.mark.parametrize("storage", ["dense", "csr"])
@pytest.mark.parametrize("d,m", [(2050, 4500), (2050, 8200), (260, 33000)])
@pytest.mark.parametrize("kernel,cnt", [("rbf", [70, 60]), ("rbf", [20, 31, 12]), ("linear", [9, 16, 17, 0, 1, 64, 33, 2, 5, 40]),
                                        ("rbf", [11] * 12), ("linear", [4] * 33)])
def test_fused_prediction_over_several_launches(capi, storage, d, m, kernel, cnt):
    """More test rows than one launch takes (4,096 of 2,050 features, some 31,000 of 260): presets and results of every slab, the
    last one shorter; test rows and support vectors on the lanes; sums by pair and by row; dense data, and CSR data that is
    worked on as dense rows."""
    rng = np.random.default_rng(m)
    n_sv = sum(cnt)
    if storage == "dense":
        SV, T = (rng.standard_normal((k, d)).astype(np.float32) for k in (n_sv, m))
        km, batch = capi.KernelMatrix(dense=_t(SV), kernel=kernel, gamma=1.0 / d), dict(dense=_t(T))
    else:
        SV, T = ((rng.random((k, d)) < 0.03).astype(np.float32) for k in (n_sv, m))
        csr = [(_t(np.ones(int(a.sum()), np.float32)), _t(np.concatenate([[0], np.cumsum((a != 0).sum(1))]).astype(np.int32)),
                _t(np.nonzero(a)[1].astype(np.int32))) for a in (SV, T)]
        km, batch = capi.KernelMatrix(csr=csr[0], d=d, kernel=kernel, gamma=1.0 / d), dict(csr=csr[1])
    _sums_case(capi, km, SV, T, kernel, 1.0 / d, cnt, len(cnt), batch)


@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 64, 65])
@pytest.mark.parametrize("storage", ["dense", "dense_sv_csr_rows", "csr"])
@pytest.mark.parametrize("nc,n_sv,d,kernel", [(2, 1, 1, "rbf"), (2, 700, 35, "rbf"), (3, 129, 4, "linear"),
                                              (32, 300, 70, "poly")])
def test_prediction_of_few_rows(capi, m, storage, nc, n_sv, d, kernel):
    """Up to eight tiles of eight rows go through one launch; sizes around its row tiles, one and several support vectors
    per block, more blocks than support vectors, features that are no multiple of four, test rows with features beyond
    the support vectors'."""
    rng = np.random.default_rng(m * 7 + nc)
    dt = d + 3                                       # the extra features count in the test rows' self dots only
    SVd = (rng.standard_normal((n_sv, d)) * (rng.random((n_sv, d)) < 0.7)).astype(np.float32)
    T = (rng.standard_normal((m, dt)) * (rng.random((m, dt)) < 0.7)).astype(np.float32)
    cnt = np.bincount(np.arange(n_sv) % nc, minlength=nc).astype(np.int32)
    coef = rng.standard_normal((nc - 1, n_sv))
    rho = rng.standard_normal(nc * (nc - 1) // 2)
    kw = dict(kernel=kernel, gamma=0.05, coef0=0.5, degree=2)
    want = P.predict_dec(P.Csr(dense=SVd), coef.reshape(-1), cnt, rho, nc, P.Csr(dense=T), **kw)

    def csr(a):
        nz = a != 0
        rp = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32)
        return _t(a[nz]), _t(rp), _t(np.nonzero(nz)[1].astype(np.int32))

    km = capi.KernelMatrix(csr=csr(SVd), d=d, **kw) if storage == "csr" else capi.KernelMatrix(dense=_t(SVd), **kw)
    batch = dict(dense=_t(T)) if storage == "dense" else dict(csr=csr(T))
    for _ in range(2):                               # the second call finds the first one's sums cleared
        dec = capi.predict_dec(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, **batch)
        assert np.max(np.abs(dec.cpu().numpy() - want)) < 1e-4 * max(1.0, np.max(np.abs(want)))
        lab = capi.predict_labels(km, _t(coef.reshape(-1)), cnt, _t(rho), nc, **batch)
        assert np.array_equal(lab.cpu().numpy(), capi.vote(dec, nc).cpu().numpy())
    km.close()


@pytest.mark.parametrize("d,fill,values", [(33, 0.3, "ones"), (256, 0.01, "ones"), (257, 0.01, "ones"), (300, 0.1, "halves"),
                                           (120, 0.1, "thirds"), (120, 0.1, "large"), (120, 0.1, "descending")])
@pytest.mark.parametrize("batch", ["ones", "thirds"])
def test_sparse_data_worked_on_as_dense_rows(capi, d, fill, values, batch):
    """CSR data that one FP16 number per entry holds exactly may go through the dense engine: the first and the last
    feature count, a fill below the line, values and orders of the entries that rule it out, batches that do. Kernel
    rows by index and by instance, decision values of 200 rows (more than the few-row launch takes)."""
    rng = np.random.default_rng(d)

    def csr(n, width, kind):
        nz = rng.random((n, width)) < fill
        rp = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32)
        col = np.nonzero(nz)[1].astype(np.int32)
        v = rng.integers(1, 8, len(col)).astype(np.float32)
        v = {"halves": v * 0.5, "thirds": v / 3, "large": v * 100}.get(kind, np.ones(len(col))).astype(np.float32)
        if kind == "descending":
            for i in range(n):
                col[rp[i]:rp[i + 1]] = col[rp[i]:rp[i + 1]][::-1].copy()
        return v, rp, col

    n, m, gamma = 301, 200, 0.05 if values != "large" else 1e-6
    sv, t = csr(n, d, values), csr(m, d + 5, batch)
    km = capi.KernelMatrix(csr=tuple(map(_t, sv)), d=d, gamma=gamma)
    assert not km.is_dense
    ids = rng.choice(n, 130, replace=False).astype(np.int32)
    want = P.kernel_rows_idx(P.Csr(csr=sv, d=d), ids, gamma=gamma)
    assert np.max(np.abs(km.get_rows(_t(ids)).cpu().numpy() - want)) < 1e-5
    want = P.kernel_rows_ins(P.Csr(csr=sv, d=d), P.Csr(csr=t, d=d + 5), gamma=gamma)
    assert np.max(np.abs(km.get_rows_instances(csr=tuple(map(_t, t))).cpu().numpy() - want)) < 1e-5
    cnt = np.array([100, 150, 51], np.int32)
    coef, rho = rng.standard_normal((2, n)), rng.standard_normal(3)
    want = P.predict_dec(P.Csr(csr=sv, d=d), coef.reshape(-1), cnt, rho, 3, P.Csr(csr=t, d=d + 5), gamma=gamma)
    dec = capi.predict_dec(km, _t(coef.reshape(-1)), cnt, _t(rho), 3, csr=tuple(map(_t, t)))
    assert np.max(np.abs(dec.cpu().numpy() - want)) < 1e-4 * max(1.0, np.max(np.abs(want)))
    km.close()
