"""The small symmetric eigensolver at the edges of its layouts: bisection groups of 7, 3 and 1 threads
(36/37 and 85/86 pairs), rows of one and several warps (32/33, 64/65, 257), clusters beside
isolated eigenvalues (a cluster is wanted whole: which members of a cut one come back is open)."""
import ctypes

import numpy as np
import pytest

from votca_gb300 import _lib

pytestmark = pytest.mark.gpu


# backward error of the reduction and the Rayleigh quotients: a few m eps |T|, |T| = 30
@pytest.mark.parametrize("m,nw", [(1, 1), (2, 2), (3, 1), (32, 8), (33, 9), (36, 36), (37, 37), (64, 20), (65, 20),
                                  (85, 85), (86, 86), (257, 3), (300, 260)])
@pytest.mark.parametrize("cluster", [False, True])
def test_lowest_pairs(m, nw, cluster):
    if cluster and nw < min(m, 3):
        pytest.skip("the cluster of three would be cut")
    rng = np.random.default_rng(m + nw)
    d = np.linspace(5.0, 30.0, m)
    if cluster:
        d[: min(m, 3)] = 5.0 + 1e-7 * np.arange(min(m, 3))
    Q = np.linalg.qr(rng.standard_normal((m, m)))[0]
    T = (Q * d) @ Q.T
    T = np.asfortranarray(0.5 * (T + T.T))
    lam, U = np.zeros(nw), np.zeros((m, nw), order="F")
    i64 = lambda x: np.array([x], dtype=np.int64).ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    p = lambda a: a.ctypes.data_as(_lib.c_dp)
    _lib.check(_lib.load().bse_small_sym_eig(1, i64(m), i64(nw), p(T), p(lam), p(U), None))
    tol = 30.0 * m * 2.0**-49
    assert np.abs(lam - d[:nw]).max() < tol
    assert np.abs(T @ U - U * lam).max() < tol
    # vectors of eigenvalues a gap apart: the backward error over the gap
    assert np.abs(U.T @ U - np.eye(nw)).max() < max(1.0, (m - 1) / 25.0) * tol
