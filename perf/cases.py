"""Performance cases: what a user of this library runs, through its public entry points.

Three kinds of work:
  solve    train one binary problem on the GPU: kernel matrix, solver, alpha / f / rho (thundersvm_b200.capi)
  predict  decision values or labels of a batch of rows against a model that is already on the GPU (capi)
  fit      the reference-named C symbols on host arrays: train a model, then predict new rows with it

Shapes and value laws are those of the repository's five benchmark configurations (thundersvm_b200/synth.py),
generated on the GPU so that preparing a case is quick:
  blobs   two clipped Gaussian blobs, few features                      (configuration 1)
  ones    CSR, a fixed number of ones per row at random columns         (configuration 2)
  pixels  class prototypes in [0, 1] plus noise, small values zeroed    (configuration 3)
  text    CSR, Zipf-distributed columns, log-normal values, unit rows   (configuration 4)
  unit    Gaussian rows scaled to length one                            (configuration 5)
"""
import ctypes
import math

import numpy as np
import torch

from thundersvm_b200 import capi

EPS = 1e-3                 # the reference's default stopping tolerance
SVM_TYPES = {"c_svc": 0, "epsilon_svr": 3}


def listed():
    return [
        # epsilon-SVR on a small table, the smallest thing people fit (through the C symbols the Python package calls)
        dict(name="fit_svr_506x13", op="fit", svm="epsilon_svr", data="blobs", n=506, d=13, m=101, classes=1, gamma=0.1,
             C=10.0),
        # ten-class one-vs-one classification of host rows, then the labels of unseen ones (configuration 3's shape)
        dict(name="fit_ovo_20000x784", op="fit", svm="c_svc", data="pixels", n=20000, d=784, m=4000, classes=10,
             gamma=0.125, C=10.0),
        # dense tables with few columns: configuration 1
        dict(name="solve_blobs_10000x20", op="solve", data="blobs", n=10000, d=20, solver="c", kernel="rbf", gamma=0.5,
             C=10.0),
        # one-hot encoded records, CSR: configuration 2
        dict(name="solve_ones_32561x123", op="solve", data="ones", n=32561, d=123, k=14, solver="c", kernel="rbf",
             gamma=0.5, C=100.0),
        # one pair of image classes, dense, an odd row count: configuration 3
        dict(name="solve_pixels_12003x784", op="solve", data="pixels", n=12003, d=784, solver="c", kernel="rbf",
             gamma=0.125, C=10.0),
        # documents, CSR with many columns: configuration 4
        dict(name="solve_text_20242x47236", op="solve", data="text", n=20242, d=47236, k=74, solver="c", kernel="rbf",
             gamma=1.0, C=100.0),
        # nu-SVC with a polynomial kernel on a ragged shape
        dict(name="solve_nu_poly_5001x61", op="solve", data="unit", n=5001, d=61, solver="nu_svc", kernel="poly",
             gamma=1.0, nu=0.3),
        # the largest training run: configuration 5's row length, half its rows
        dict(name="solve_unit_200000x2000", op="solve", data="unit", n=200000, d=2000, solver="c", kernel="rbf",
             gamma=0.5, C=1.0),
        # a service that scores single rows as they arrive
        dict(name="predict_1row_3001x100", op="predict", data="unit", n_sv=3001, d=100, m=1, classes=2, out="dec",
             gamma=0.5),
        # labels of a ten-class test set: configuration 3's prediction
        dict(name="predict_ovo_10000x784", op="predict", data="pixels", n_sv=8003, d=784, m=10000, classes=10,
             out="labels", gamma=0.125),
        # CSR model, CSR test rows: configuration 2's prediction
        dict(name="predict_ones_16281x123", op="predict", data="ones", n_sv=12001, d=123, k=14, m=16281, classes=2,
             out="dec", gamma=0.5),
        # the largest prediction: configuration 5's test set against a model of half its training rows
        dict(name="predict_unit_100000x2000", op="predict", data="unit", n_sv=200000, d=2000, m=100000, classes=2,
             out="labels", gamma=0.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: every kind, storage and option of the listed ones, sizes over the whole range."""
    op = rng.choice(["fit", "solve", "solve", "solve", "predict", "predict"])
    if op == "fit":
        if rng.random() < 0.5:
            n = _log_int(rng, 150, 3000)
            return dict(op=op, svm="epsilon_svr", data="blobs", n=n, d=rng.randint(4, 40), m=max(10, n // 5), classes=1,
                        gamma=0.1, C=10.0)
        n = _log_int(rng, 1000, 16000)
        return dict(op=op, svm="c_svc", data="pixels", n=n, d=_log_int(rng, 50, 784), m=max(50, n // 5),
                    classes=rng.randint(2, 10), gamma=0.125, C=10.0)
    data = rng.choice(["blobs", "ones", "pixels", "text", "unit"])
    if op == "solve":
        case = dict(op=op, data=data, solver="c", kernel="rbf", gamma=0.5, C=10.0)
        if data == "blobs":
            case.update(n=_log_int(rng, 200, 16000), d=rng.randint(4, 64))
        elif data == "ones":
            case.update(n=_log_int(rng, 1000, 33000), d=rng.randint(60, 200), k=rng.randint(8, 20), C=100.0)
        elif data == "pixels":
            case.update(n=_log_int(rng, 500, 15000), d=_log_int(rng, 50, 800), gamma=0.125)
        elif data == "text":
            case.update(n=_log_int(rng, 1000, 20000), d=_log_int(rng, 5000, 50000), k=rng.randint(30, 90), gamma=1.0,
                        C=100.0)
        elif rng.random() < 0.4:
            case.update(n=_log_int(rng, 500, 6000), d=rng.randint(10, 100), solver="nu_svc", kernel="poly", gamma=1.0,
                        nu=0.3)
        else:
            case.update(n=_log_int(rng, 1000, 120000), d=_log_int(rng, 40, 2000), C=1.0)
        return case
    classes = rng.choice([2, 2, rng.randint(3, 10)])
    case = dict(op=op, data=data, classes=classes, out=rng.choice(["dec", "labels"]), gamma=0.5)
    case["m"] = _log_int(rng, 1, 20000)
    case["n_sv"] = _log_int(rng, 20 * classes, 40000 if data == "unit" else 12000)
    if data == "ones":
        case.update(d=rng.randint(60, 200), k=rng.randint(8, 20))
    elif data == "text":
        case.update(d=_log_int(rng, 5000, 50000), k=rng.randint(30, 90), gamma=1.0)
    elif data == "pixels":
        case.update(d=_log_int(rng, 50, 800), gamma=0.125)
    else:
        case.update(d=rng.randint(4, 64) if data == "blobs" else _log_int(rng, 40, 2000))
    return case


# ---- data -----------------------------------------------------------------------------------------------
def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _dense_rows(data, n, d, classes, law, rows):
    """-> X [n, d] float32, class of every row, score (blobs / unit: position relative to a random hyperplane).
    `law` fixes the prototypes and the hyperplane, `rows` the rows drawn."""
    if data == "pixels":
        on = torch.rand(classes, d, generator=law, device="cuda") < 0.19
        proto = torch.where(on, 0.5 + 0.5 * torch.rand(classes, d, generator=law, device="cuda"), torch.zeros((), device="cuda"))
        cls = torch.randint(0, classes, (n,), generator=rows, device="cuda")
        X = (proto[cls] + 0.1 * torch.randn(n, d, generator=rows, device="cuda")).clamp_(0.0, 1.0)
        X[X < 0.05] = 0.0
        return X, cls, None
    w = torch.randn(d, generator=law, device="cuda")
    X = torch.randn(n, d, generator=rows, device="cuda")
    if data == "blobs":
        cls = (torch.rand(n, generator=rows, device="cuda") < 0.4).long()
        X += 0.5 * (2.0 * cls.float() - 1.0)[:, None]
        X.clamp_(-3.0, 3.0)
    else:
        X /= X.square().sum(1, keepdim=True).sqrt()
        cls = None
    return X, cls, X @ w


def _csr_rows(data, n, d, k, law, rows):
    """-> (val, row_ptr, col), score of a random sparse teacher."""
    if data == "ones":
        col = torch.rand(n, d, generator=rows, device="cuda").argsort(1)[:, :k].sort(1).values.int()
        val = torch.ones(n * k, device="cuda")
        row_ptr = torch.arange(0, n * k + 1, k, dtype=torch.int32, device="cuda")
        score = torch.randn(d, generator=law, device="cuda")[col.long()].sum(1)
        return (val, row_ptr, col.reshape(-1).contiguous()), score
    # text: Poisson(k) >= 1 distinct columns per row out of Zipf(1.1) draws
    p = torch.arange(1, d + 1, dtype=torch.float64, device="cuda").pow(-1.1)
    cdf = (p / p.sum()).cumsum(0).float()
    wide = 2 * k + 8
    col = torch.searchsorted(cdf, torch.rand(n, wide, generator=rows, device="cuda")).clamp_(max=d - 1).sort(1).values
    want = torch.poisson(torch.full((n, 1), float(k), device="cuda"), generator=rows).clamp_(min=1)
    first = torch.ones_like(col, dtype=torch.bool)
    first[:, 1:] = col[:, 1:] != col[:, :-1]
    order = torch.where(first, torch.rand(n, wide, generator=rows, device="cuda"), torch.full((), 2.0, device="cuda"))
    keep = first & (order.argsort(1).argsort(1) < want)
    val = torch.randn(n, wide, generator=rows, device="cuda").exp() * keep
    val /= val.square().sum(1, keepdim=True).sqrt()
    teacher = torch.randn(d, generator=law, device="cuda")
    score = (val * teacher[col]).sum(1)
    row_ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = keep.sum(1).cumsum(0)
    return (val[keep].contiguous(), row_ptr, col[keep].int().contiguous()), score


def _labels(cls, score, positive, flips, rows, missed=0.0):
    """+1 / -1: the given class, or the top `positive` share of the score; a share of all labels is flipped, and a share
    of the positive ones is missed."""
    up = cls == 0 if cls is not None else score > score.quantile(1.0 - positive)
    noise = torch.rand(up.numel(), generator=rows, device="cuda")
    return torch.where(up ^ ((noise < flips) | (up & (noise < missed))), 1, -1).to(torch.int32)


def _is_csr(case):
    return case["data"] in ("ones", "text")


# ---- prepare --------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"solve": _prepare_solve, "predict": _prepare_predict, "fit": _prepare_fit}[case["op"]](case, seed)


def _prepare_solve(case, seed):
    law, rows = _generator(seed, 1), _generator(seed, 2)
    n, d, data = case["n"], case["d"], case["data"]
    if _is_csr(case):
        csr, score = _csr_rows(data, n, d, case["k"], law, rows)
        mats = dict(csr=csr, d=d)
        y = _labels(None, score, 0.24 if data == "ones" else 0.52, 0.02, rows)
    else:
        X, cls, score = _dense_rows(data, n, d, 2, law, rows)
        mats = dict(dense=X)
        flips = {"blobs": 0.05, "pixels": 0.0, "unit": 0.1}[data]
        y = _labels(cls, score, 0.4, flips, rows, missed=0.04 if data == "pixels" else 0.0)
    return dict(case=case, mats=mats, y=y, ws=capi.working_set_size(n, d))


def _prepare_predict(case, seed):
    law, rows, coefs = _generator(seed, 1), _generator(seed, 2), _generator(seed, 3)
    n_sv, m, d, classes = case["n_sv"], case["m"], case["d"], case["classes"]
    if _is_csr(case):
        sv, _ = _csr_rows(case["data"], n_sv, d, case["k"], law, rows)
        test, _ = _csr_rows(case["data"], m, d, case["k"], law, rows)
        km = capi.KernelMatrix(csr=sv, d=d, gamma=case["gamma"])
        batch = dict(csr=test)
    else:
        # model and test rows of the same prototypes: one draw, split
        X, _, _ = _dense_rows(case["data"], n_sv + m, d, classes, law, rows)
        km = capi.KernelMatrix(dense=X[:n_sv].clone(), gamma=case["gamma"])
        batch = dict(dense=X[n_sv:].clone())
    count = [n_sv // classes + (1 if c < n_sv % classes else 0) for c in range(classes)]
    # signs as a trained model has them: positive for the first class of a pair, negative for the second
    coef = torch.rand(classes - 1, n_sv, generator=coefs, dtype=torch.float64, device="cuda")
    owner = torch.repeat_interleave(torch.arange(classes, device="cuda"), torch.tensor(count, device="cuda"))
    other = torch.arange(classes - 1, device="cuda")[:, None]
    coef = torch.where(other >= owner[None, :], coef, -coef).contiguous()
    rho = torch.rand(classes * (classes - 1) // 2, generator=coefs, dtype=torch.float64, device="cuda") - 0.5
    return dict(case=case, km=km, batch=batch, count=count, coef=coef, rho=rho)


def _prepare_fit(case, seed):
    law, rows = _generator(seed, 1), _generator(seed, 2)
    n, m, d = case["n"], case["m"], case["d"]
    X, cls, score = _dense_rows(case["data"], n + m, d, case["classes"], law, rows)
    if case["svm"] == "c_svc":
        # two labels in a hundred are wrong; the first rows hold one of every class, in order
        wrong = torch.rand(n + m, generator=rows, device="cuda") < 0.02
        y = torch.where(wrong, torch.randint(0, case["classes"], (n + m,), generator=rows, device="cuda"), cls)
        y[:case["classes"]] = torch.arange(case["classes"], device="cuda")
    else:
        y = 3.0 + 0.3 * score + torch.sin(X[:, 0]) + 0.1 * torch.randn(n + m, generator=rows, device="cuda")
    return dict(case=case, X=X[:n].cpu().numpy(), y=y[:n].float().cpu().numpy(), T=X[n:].cpu().numpy(), lib=_symbols())


def _symbols():
    """The reference-named C symbols of the library, as the reference's Python package declares them."""
    lib = ctypes.CDLL(capi.LIB_PATH)
    f, i, vp = ctypes.c_float, ctypes.c_int, ctypes.c_void_p
    lib.model_new.restype, lib.model_new.argtypes = vp, [i]
    lib.model_free.argtypes = [vp]
    lib.dense_model_scikit.argtypes = [i, i, vp, vp, i, i, i, f, f, f, f, f, f, i, i, vp, vp, i, i, i, i, i, vp, vp, vp, vp]
    lib.dense_predict.argtypes = [i, i, vp, vp, vp, i]
    lib.get_rho.argtypes = [vp, i, vp]
    return lib


# ---- run ------------------------------------------------------------------------------------------------
def run(state):
    return {"solve": _run_solve, "predict": _run_predict, "fit": _run_fit}[state["case"]["op"]](state)


def _run_solve(state):
    case, y = state["case"], state["y"]
    km = capi.KernelMatrix(kernel=case["kernel"], gamma=case["gamma"], coef0=1.0 if case["kernel"] == "poly" else 0.0,
                           **state["mats"])
    if case["solver"] == "c":
        C = case["C"]
        alpha = torch.zeros(y.numel(), dtype=torch.float64, device="cuda")
        f = -y.to(torch.float64)
    else:
        # nu-SVC starts with nu * n / 2 of alpha in each class, filled from the front
        C = 1.0
        each = case["nu"] * y.numel() / 2
        pos = y > 0
        alpha = torch.where(pos, each - (pos.cumsum(0) - 1), each - ((~pos).cumsum(0) - 1)).to(torch.float64).clamp_(0.0, 1.0)
        f = torch.zeros(y.numel(), dtype=torch.float64, device="cuda")
    rho, _ = capi.smo_solve(km, y, alpha, f, EPS, C, C, state["ws"], solver=case["solver"])
    km.close()
    return dict(alpha=alpha, f=f, rho=rho)


def _run_predict(state):
    call = capi.predict_dec if state["case"]["out"] == "dec" else capi.predict_labels
    return call(state["km"], state["coef"], state["count"], state["rho"], state["case"]["classes"], **state["batch"])


def _run_fit(state):
    case, lib, X, y, T = state["case"], state["lib"], state["X"], state["y"], state["T"]
    svm = SVM_TYPES[case["svm"]]
    pairs = max(1, case["classes"] * (case["classes"] - 1) // 2)
    n_features, n_classes, ok = (np.zeros(1, np.int32) for _ in range(3))
    out, rho = np.zeros(case["m"], np.float32), np.zeros(pairs, np.float32)
    model = lib.model_new(svm)
    lib.dense_model_scikit(X.shape[0], X.shape[1], X.ctypes.data, y.ctypes.data, svm, 2, 3, case["gamma"], 0.0, case["C"],
                           0.5, 0.1, EPS, 0, 0, None, None, 0, -1, -1, -1, 0, n_features.ctypes.data,
                           n_classes.ctypes.data, ok.ctypes.data, model)
    lib.get_rho(rho.ctypes.data, pairs, model)
    lib.dense_predict(T.shape[0], T.shape[1], T.ctypes.data, model, out.ctypes.data, 0)
    lib.model_free(model)
    return dict(rho=rho, predicted=out.astype(np.int32) if case["svm"] == "c_svc" else out)


# ---- what the work is -----------------------------------------------------------------------------------
def work(case):
    """Bytes: every input and output once. Operations: the kernel values that the result depends on - every test row
    against every support vector; in training, every instance against the half of them that a typical run looks at -
    times the multiply-adds of one value (sparse rows: one per stored entry)."""
    per_value = 2.0 * (case["k"] if _is_csr(case) else case["d"])
    row_bytes = 8.0 * case["k"] if _is_csr(case) else 4.0 * case["d"]
    if case["op"] == "predict":
        pairs = case["classes"] * (case["classes"] - 1) // 2
        out = case["m"] * (8.0 * pairs if case["out"] == "dec" else 4.0)
        return dict(bytes=(case["n_sv"] + case["m"]) * row_bytes + 8.0 * case["n_sv"] * (case["classes"] - 1) + out,
                    flops=case["n_sv"] * float(case["m"]) * per_value)
    n = case["n"]
    if case["op"] == "solve":
        return dict(bytes=n * (row_bytes + 4.0 + 16.0), flops=n * (n / 2.0) * per_value)
    # every class pair has 2 n / classes instances; SVR duplicates its n instances
    problems = max(1, case["classes"] * (case["classes"] - 1) // 2)
    size = 2.0 * n / max(1, case["classes"])
    return dict(bytes=(n + case["m"]) * (row_bytes + 4.0), flops=problems * size * (size / 2.0) * per_value)


def tolerance(case):
    """Kernel values are FP32, sums of them FP64: predictions agree to the FP32 rounding of the values. A solver stops at
    a violation of EPS = 1e-3, so two correct solvers (or one, with gamma changed in its last digit) agree to about that,
    and a single alpha of nearly exchangeable instances to less."""
    if case["op"] == "predict":
        return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
    if case["op"] == "solve":
        return {"rel": 2e-2, "max": 0.3}
    return {"rel": 3e-3, "max": 0.05, "differ": 2e-3}
