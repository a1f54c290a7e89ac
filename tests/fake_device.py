"""Runs the library's host code in a child process on a stand-in for the CUDA runtime (fake_cudart.cpp): memory with a
limit, kernels that do nothing, counters. For what cannot be arranged on a real device: one that is full, and proof of what
is waited for. Kernels' results are not looked at."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, %r)
F = C.CDLL(None)
for name in ("fake_set_free",): getattr(F, name).argtypes = [C.c_size_t]
for name in ("fake_used", "fake_largest_refused"): getattr(F, name).restype = C.c_size_t
for name in ("fake_launches", "fake_device_waits", "fake_stream_waits"): getattr(F, name).restype = C.c_longlong
L = C.CDLL(%r)
L.tsvm_last_error.restype = C.c_char_p
L.tsvm_km_destroy.argtypes = L.tsvm_solver_destroy.argtypes = [C.c_void_p]
L.tsvm_km_nnz.restype = C.c_longlong
L.tsvm_km_nnz.argtypes = [C.c_void_p]
OK, OOM, MB = 0, 3, 1 << 20
HOST, DEVICE, RBF = 0, 1, 2
def p(a): return C.c_void_p(a.ctypes.data)
def dense(X, loc=HOST):
    h = C.c_void_p()
    return L.tsvm_km_create_dense(p(X), X.shape[0], X.shape[1], X.shape[1], loc, RBF, 3, C.c_float(0.5), C.c_float(0), None, C.byref(h)), h
def csr(n, d, per_row, loc=HOST):
    rp = np.arange(0, n * per_row + 1, per_row, dtype=np.int32)
    col = np.tile(np.arange(per_row, dtype=np.int32), n)
    val = np.ones(n * per_row, np.float32)
    h = C.c_void_p()
    s = L.tsvm_km_create_csr(p(val), p(rp), p(col), n, d, loc, RBF, 3, C.c_float(0.5), C.c_float(0), None, C.byref(h))
    return s, h, (val, rp, col)
def solver(h, n, ws=1024):
    y, a, f = np.ones(n, np.int32), np.zeros(n), np.zeros(n)
    s = C.c_void_p()
    r = L.tsvm_solver_create(h, 0, p(y), p(a), p(f), C.c_double(1e-3), C.c_double(1), C.c_double(1), ws, None, C.byref(s))
    return r, s, (y, a, f)
def check(status, want=OK): assert status == want, (status, L.tsvm_last_error())
""" % (HERE, os.path.join(ROOT, "thundersvm_b200", "libthundersvm_b200.so"))


def compile_runtime(out_dir):
    path = os.path.join(str(out_dir), "fake_cudart.so")
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-I/usr/local/cuda/include",
                           os.path.join(HERE, "fake_cudart.cpp"), "-o", path])
    return path


def run_child(runtime, command):
    env = dict(os.environ, LD_PRELOAD=runtime, CUDA_VISIBLE_DEVICES="", OMP_NUM_THREADS="2")
    env.pop("TSVM_ROW_CACHE_MB", None)
    r = subprocess.run(command, env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    return r.stdout


def run_python(runtime, body):
    return run_child(runtime, [sys.executable, "-c", PRELUDE + body])
