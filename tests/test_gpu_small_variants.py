"""The small dense solvers of the Davidson iteration in both of their forms (with divisions: split-precision
solves, lockstep batches and the solvers' own entry points; without: FP64 solves) at the edges of their
layouts, through the same checks: the symmetric eigensolver, the harmonic-Ritz solver and the Cholesky QR."""
import ctypes

import numpy as np
import pytest

import native
from votca_gb300 import _lib

pytestmark = pytest.mark.gpu

p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
i64 = ctypes.c_int64


def _sym(T, nw, fast):
    L = native.load()
    m = T.shape[0]
    lam, U = np.zeros(nw), np.zeros((m, nw), order="F")
    assert L.shim_sym_eig(p(T), i64(m), i64(nw), fast, p(lam), p(U)) == 0, L.shim_last_error()
    return lam, U


def _gen(T, B, nw, fast):
    L = native.load()
    m = T.shape[0]
    lam, U, sel = np.zeros(nw), np.zeros((m, nw), order="F"), ctypes.c_int()
    assert L.shim_gen_eig(p(T), p(B), i64(m), i64(nw), fast, p(lam), p(U), ctypes.byref(sel)) == 0, L.shim_last_error()
    return lam, U, sel.value


# tolerances as in test_gpu_sym_eig_sizes.py and test_gpu_harmonic_ritz_sizes.py
@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("m,nw", [(1, 1), (2, 2), (3, 1), (32, 8), (33, 9), (37, 37), (64, 20), (65, 20), (86, 86), (257, 3)])
def test_symmetric(m, nw, fast):
    rng = np.random.default_rng(m + nw)
    d = np.linspace(5.0, 30.0, m)
    Q = np.linalg.qr(rng.standard_normal((m, m)))[0]
    T = (Q * d) @ Q.T
    T = np.asfortranarray(0.5 * (T + T.T))
    lam, U = _sym(T, nw, fast)
    tol = 30.0 * m * 2.0**-49
    assert np.abs(lam - d[:nw]).max() < tol
    assert np.abs(T @ U - U * lam).max() < tol
    assert np.abs(U.T @ U - np.eye(nw)).max() < max(1.0, (m - 1) / 25.0) * tol


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("m,nw", [(1, 1), (2, 2), (31, 31), (60, 33), (97, 4), (98, 4), (128, 40), (129, 3)])
def test_pencil(m, nw, fast):
    rng = np.random.default_rng(m)
    d = np.linspace(1.0, 3.0, m)
    Q = np.linalg.qr(rng.standard_normal((m, m)))[0]
    T = (Q * d) @ Q.T
    T = np.asfortranarray(0.5 * (T + T.T))
    B = np.asfortranarray(T @ T)
    lam, U, sel = _gen(T, B, nw, fast)
    assert sel == nw
    np.testing.assert_allclose(lam, d[:nw], rtol=0, atol=1e-10)
    assert np.abs(T @ U - U * lam).max() < 1e-10


def test_entry_points_divide():
    """bse_small_sym_eig and bse_small_gen_eig: the variants with divisions, to the last bit."""
    L = _lib.load()
    rng = np.random.default_rng(5)
    m, nw = 40, 12
    T = rng.standard_normal((m, m))
    T = np.asfortranarray(T + T.T)
    one = lambda x: np.array([x], dtype=np.int64).ctypes.data_as(ctypes.POINTER(i64))
    dp = lambda a: a.ctypes.data_as(_lib.c_dp)
    lam, U = np.zeros(nw), np.zeros((m, nw), order="F")
    _lib.check(L.bse_small_sym_eig(1, one(m), one(nw), dp(T), dp(lam), dp(U), None))
    ref = _sym(T, nw, 0)
    np.testing.assert_array_equal(lam, ref[0])
    np.testing.assert_array_equal(U, ref[1])
    B = np.asfortranarray(T @ T + 40 * np.eye(m))
    sel = i64()
    _lib.check(L.bse_small_gen_eig(m, nw, dp(T), dp(B), dp(lam), dp(U), ctypes.byref(sel)))
    ref = _gen(T, B, nw, 0)
    np.testing.assert_array_equal(lam, ref[0])
    np.testing.assert_array_equal(U, ref[1])


def _cholqr(G, n0, fast):
    L = native.load()
    nb = G.shape[0]
    R, ok, flag = np.zeros((nb, nb), order="F"), ctypes.c_int(7), ctypes.c_int(0)
    assert L.shim_cholqr(p(np.asfortranarray(G)), nb, p(n0), 1, fast, p(R), ctypes.byref(ok), ctypes.byref(flag)) == 0
    return R, ok.value, flag.value


# G = X^T X of unit columns: with Q = X R^-1, the Gram matrix of Q is off by a few nb eps cond(X)^2
@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("nb", [1, 2, 3, 8, 17, 31, 32, 33, 63, 64])
def test_cholesky_qr(nb, fast):
    rng = np.random.default_rng(nb)
    X = rng.standard_normal((6 * nb + 3, nb))
    X /= np.linalg.norm(X, axis=0)
    R, ok, flag = _cholqr(X.T @ X, np.ones(nb), fast)
    assert (ok, flag) == (1, 0)
    assert np.all(np.tril(R, -1) == 0.0)
    Q = X @ R
    assert np.abs(Q.T @ Q - np.eye(nb)).max() < 16 * nb * 2.0**-52 * np.linalg.cond(X) ** 2


# A pivot below 1e-10 of its diagonal is left to the column-by-column Gram-Schmidt, which decides whether the
# column is dependent: the factorisation itself must not (an exact zero is cancellation, not a norm).
@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("off", [0.0, 2.0**-48, -(2.0**-50)])
def test_small_pivot_is_not_a_verdict(off, fast):
    G = np.eye(3)
    G[1, 2] = G[2, 1] = 1.0
    G[2, 2] = 1.0 + off
    _, ok, flag = _cholqr(G, np.ones(3), fast)
    assert (ok, flag) == (0, 0)


# beyond it the column is there, but of no norm: dependent
@pytest.mark.parametrize("fast", [0, 1])
def test_lost_norm_is_reported(fast):
    _, ok, flag = _cholqr(np.eye(3), np.array([1.0, 1.0, 1e13]), fast)
    assert (ok, flag) == (1, 1)
