"""The harmonic-Ritz solver at the edges of its layouts: matrices in shared memory or not (m = 97, 98),
the parallel inverse iteration's row registers (m = 128, 129), more vectors than lanes, and
eigenvalues close enough to be a cluster beside isolated ones."""
import ctypes

import numpy as np
import pytest

from votca_gb300 import _lib

pytestmark = pytest.mark.gpu


# backward errors are a few m eps |T| (|T| = 3, cond(B) = 9): 1e-10 leaves a factor of 1000 at m = 129
@pytest.mark.parametrize("m,nw", [(1, 1), (2, 2), (31, 31), (60, 33), (97, 4), (98, 4), (128, 40), (129, 3)])
@pytest.mark.parametrize("cluster", [False, True])
def test_symmetric_pencil(m, nw, cluster):
    rng = np.random.default_rng(m)
    d = np.linspace(1.0, 3.0, m)
    if cluster and m >= 3:
        d[1] = d[0] + 1e-11
    Q = np.linalg.qr(rng.standard_normal((m, m)))[0]
    T = (Q * d) @ Q.T
    T = np.asfortranarray(0.5 * (T + T.T))
    B = np.asfortranarray(T @ T)
    lam, U, sel = np.zeros(nw), np.zeros((m, nw), order="F"), ctypes.c_int64()
    p = lambda a: a.ctypes.data_as(_lib.c_dp)
    L = _lib.load()
    _lib.check(L.bse_small_gen_eig(m, nw, p(T), p(B), p(lam), p(U), ctypes.byref(sel)))
    assert sel.value == nw
    np.testing.assert_allclose(lam, d[:nw], rtol=0, atol=1e-10)
    np.testing.assert_allclose(np.linalg.norm(U, axis=0), 1.0, rtol=0, atol=1e-12)
    # vectors of isolated eigenvalues; a cluster spans its subspace (here an eigenvector each)
    assert np.abs(T @ U - U * lam).max() < 1e-10
    for c in range(2 if cluster and m >= 3 else 0, nw):
        assert abs(abs(Q[:, c] @ U[:, c]) - 1.0) < 1e-10
