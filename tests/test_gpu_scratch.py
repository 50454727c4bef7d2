"""Scratch of the tensor-core FP64 products and of calls without a handle: what stays allocated after
a call, and products cut into chunks of rows and of batches."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import native
from votca_gb300 import screening

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _product(v, A, B, C, alpha=1.0, beta=0.0, budget=3 << 29):
    L = native.load()
    taken, keep = ctypes.c_int(), ctypes.c_int64()
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    n = lambda a: ctypes.c_int64(a.size)
    v = np.array(v, dtype=np.int64)
    assert L.shim_oz_dgemm(p(v), p(A), n(A), p(B), n(B), p(C), n(C), ctypes.c_double(alpha), ctypes.c_double(beta),
                           ctypes.c_int64(budget), 2000000, ctypes.byref(taken),
                           ctypes.byref(keep)) == 0, L.shim_last_error()
    return taken.value, keep.value


def _pool():
    r, t = ctypes.c_uint64(), ctypes.c_uint64()
    assert native.load().shim_pool_state(ctypes.byref(r), ctypes.byref(t)) == 0
    return r.value, t.value


def test_no_room_for_the_planes():
    """The FMA kernel takes over: nothing of the other path may stay allocated beside it, nor what the
    pool reserved for the attempt."""
    L = native.load()
    before = _pool()[0]
    taken, keep = ctypes.c_int(1), ctypes.c_int64(-1)
    assert L.shim_oz_no_room(ctypes.byref(taken), ctypes.byref(keep)) == 0, L.shim_last_error()
    assert (taken.value, keep.value) == (0, 0)
    assert _pool()[0] <= before + 1024 * MB


def test_large_planes_are_given_back():
    """20480 x 1024 times 1024 x 64: 294 MB of planes; a workspace keeps no more than 128 MB."""
    M, N, K = 20480, 64, 1024
    rng = np.random.default_rng(2)
    A, B, C = rng.standard_normal(M * K), rng.standard_normal(K * N), np.zeros(M * N)
    taken, keep = _product([M, N, K, 1, 1, 1, M, 0, 0, 1, K, 0, 0, 1, M, 0, 0], A, B, C)
    assert taken == 1 and keep <= 128 * MB
    rows = rng.integers(0, M, 16)
    ref = A.reshape(K, M)[:, rows].T.astype(np.longdouble) @ B.reshape(N, K).T.astype(np.longdouble)
    a, b = np.abs(A.reshape(K, M)[:, rows].T), np.abs(B.reshape(N, K).T)
    bound = K * 2.0**-53 * a.max(axis=1)[:, None] * b.max(axis=0)[None, :]
    assert np.all(np.abs(C.reshape(N, M)[:, rows].T - ref) <= bound + 2.0**-52 * np.abs(ref))


# bytes of planes per row: 14 Kp; budgets of some row tiles (of the longer side, which the plan makes the
# rows) and of one and two batches; K of one and of several exponent segments (256), runs (1024)
# and K splits
@pytest.mark.parametrize("K", [224, 257, 1100])
@pytest.mark.parametrize("M,N,batch,rows", [(130, 2600, 1, 900), (300, 2100, 1, 700), (260, 130, 7, 600), (300, 257, 5, 310)])
def test_chunks(M, N, batch, rows, K):
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((batch, M, K)), rng.standard_normal((batch, K, N))
    # every row and column its own exponent, also in reused tables
    A *= 2.0 ** rng.integers(-30, 30, (batch, M, 1))
    B *= 2.0 ** rng.integers(-30, 30, (batch, 1, N))
    C = rng.standard_normal((batch, M, N))
    C0 = C.copy()
    budget = rows * 14 * ((K + 31) // 32 * 32)
    ab, bb = (M * K, K * N) if batch > 1 else (0, 0)
    taken, _ = _product([M, N, K, batch, 1, K, 1, ab, 0, N, 1, bb, 0, N, 1, M * N, 0], A, B, C, -2.0, 0.5, budget)
    assert taken == 1
    ref = -2.0 * (A @ B) + 0.5 * C0  # itself a chain of K terms
    bound = 2.0 * K * 2.0**-53 * (np.abs(A).max(axis=2)[:, :, None] * np.abs(B).max(axis=1)[:, None, :]
                                  + np.abs(A) @ np.abs(B))
    assert np.all(np.abs(C - ref) <= bound + 2.0**-51 * (np.abs(ref) + np.abs(C0)))


def test_calls_without_a_handle_leave_the_handles_pool_alone():
    L = native.load()
    assert L.shim_pool_hold(ctypes.c_int64(1280 * MB), ctypes.c_int64(512 * MB)) == 0
    before = _pool()
    assert before[0] >= 1792 * MB
    a = np.eye(96) * 2.0
    np.testing.assert_allclose(screening.cholesky_inverse(a), 0.5 * np.eye(96), rtol=1e-15)
    after = _pool()
    assert L.shim_pool_release() == 0
    assert after == before


def test_calls_without_a_handle_leave_the_default_threshold():
    """In a process of its own, without any handle."""
    code = """
import ctypes, numpy as np, native
from votca_gb300 import screening
screening.cholesky_inverse(np.eye(300) * 2.0)
r, t = ctypes.c_uint64(), ctypes.c_uint64()
assert native.load().shim_pool_state(ctypes.byref(r), ctypes.byref(t)) == 0
print("pool", r.value, t.value)
"""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split()[-3:] == ["pool", "0", "0"], r.stdout


# n below, at and above the blocks (64) and their pairs, with a short last pair
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 190, 257, 449, 640])
def test_cholesky_inverse_in_place(n):
    """Without room for a third matrix, what the call took before the factor had one of its own."""
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n + 20))
    A = np.asfortranarray(B @ B.T / n + np.eye(n))
    W = np.zeros((n, n), order="F")
    L = native.load()
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert L.shim_cholesky_inverse_in_place(ctypes.c_int64(n), p(A), p(W)) == 0, L.shim_last_error()
    # n eps |W| |A| |W| for the factorisation and the products each, |A| < 8, |W| <= 1
    assert np.abs(W - np.linalg.inv(A)).max() < 16 * 8 * n * 2.0**-53
    np.testing.assert_allclose(W, screening.cholesky_inverse(A), rtol=0, atol=16 * 8 * n * 2.0**-53)
