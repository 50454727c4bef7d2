"""The small dense solvers of the Davidson iteration in both of their forms (with divisions: split-precision
solves; without: FP64 solves) at the edges of their layouts, through the same checks: the Cholesky QR."""
import ctypes

import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu

p = lambda a: a.ctypes.data_as(ctypes.c_void_p)


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
