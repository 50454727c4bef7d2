"""FP64 products: the FMA kernel's tiles (small operators), and the products that run as exact digit products on the tensor cores (csrc/oz_gemm.cu), through
the dense operator (C = A X at any size) and the auxiliary-metric product (a batched form).

Bound: an element is rounded to 55 bits below its run's largest element, |dx| <= 2^-55 max|x|, so
a term a b is off by at most 2^-54 max|a| max|b| (the dropped digit pairs add 15 2^-64), a sum of K
terms by K times that, and the result is rounded to FP64 once per K split."""
import numpy as np
import pytest

from votca_gb300 import bse_operator as bo
from votca_gb300 import threecenter

pytestmark = pytest.mark.gpu


def _bound(A, X):
    ma = np.abs(A).max(axis=1)[:, None]
    mx = np.abs(X).max(axis=0)[None, :]
    return A.shape[1] * 2.0**-53 * ma * mx


def _exact(A, X):
    return A.astype(np.longdouble) @ X.astype(np.longdouble)


# n and k around the FMA kernel's tiles (16, 32, 64) and its K step (16) and splits; its error is
# that of a K-term chain, K 2^-53 sum |a||x|
@pytest.mark.parametrize("n", [1, 15, 17, 33, 48, 65, 100, 129])
@pytest.mark.parametrize("k", [1, 16, 17, 33, 65])
def test_fma_tiles(n, k):
    rng = np.random.default_rng(100 * n + k)
    A, X = rng.standard_normal((n, n)), rng.standard_normal((n, k))
    op = bo.DenseGpuOperator(A)
    Y = op.matmul(X)
    op.close()
    err = np.abs(Y - _exact(A, X)).astype(np.float64)
    assert np.all(err <= n * 2.0**-53 * (np.abs(A) @ np.abs(X)) + 2.0**-52 * np.abs(Y))


# n around the tile (128, 64), stage (32), drain (256) and run (1024) sizes
@pytest.mark.parametrize("n,k", [(512, 1), (513, 63), (639, 64), (641, 65), (1023, 17), (1025, 129), (2081, 5)])
@pytest.mark.parametrize("kind", ["gauss", "graded", "unit"])
def test_dense_product(n, k, kind):
    rng = np.random.default_rng(n + k)
    A, X = rng.standard_normal((n, n)), rng.standard_normal((n, k))
    if kind == "graded":
        A *= 10.0 ** rng.uniform(-9, 0, A.shape)
        X *= 10.0 ** rng.uniform(-9, 0, X.shape)
        A *= 2.0 ** rng.integers(-200, 200, (n, 1))
        X *= 2.0 ** rng.integers(-200, 200, (1, k))
        A[7] = 0.0
    if kind == "unit":
        X[:] = 0.0
        X[rng.integers(0, n, k), np.arange(k)] = 1.0
    op = bo.DenseGpuOperator(A)
    Y = op.matmul(X)
    op.close()
    err = np.abs(Y - _exact(A, X)).astype(np.float64)
    assert np.all(err <= _bound(A, X) + 2.0**-52 * np.abs(Y))
    if kind == "unit":  # single terms survive to the last bit of the run's window
        assert np.abs(Y - A @ X).max() <= 2.0**-55 * np.abs(A).max()


def test_special_values():
    rng = np.random.default_rng(3)
    n, k = 700, 70
    A, X = rng.standard_normal((n, n)), rng.standard_normal((n, k))
    A[5, 9], A[11, 3] = np.inf, np.nan
    X[2, 4], X[600, 33] = -np.inf, 1e-310
    op = bo.DenseGpuOperator(A)
    Y = op.matmul(X)
    op.close()
    with np.errstate(invalid="ignore"):
        ref = A @ X
    np.testing.assert_array_equal(np.isnan(Y), np.isnan(ref))
    np.testing.assert_array_equal(np.isinf(Y), np.isinf(ref))
    f = np.isfinite(ref)
    np.testing.assert_array_equal(Y[np.isinf(ref)], ref[np.isinf(ref)])
    np.testing.assert_allclose(Y[f], ref[f], rtol=0, atol=n * 2.0**-52 * np.abs(A[np.isfinite(A)]).max() * 6)


def test_exponent_range():
    """Values near the ends of the FP64 range give what the FMA chain gives."""
    rng = np.random.default_rng(4)
    n, k = 640, 64
    A, X = rng.standard_normal((n, n)) * 1e290, rng.standard_normal((n, k)) * 1e-290
    op = bo.DenseGpuOperator(A)
    Y = op.matmul(X)
    op.close()
    err = np.abs(Y - _exact(A, X)).astype(np.float64)
    assert np.all(err <= _bound(A, X) + 2.0**-52 * np.abs(Y))


@pytest.mark.parametrize("nmo,naux", [(33, 200), (65, 257)])
def test_batched_product(nmo, naux):
    rng = np.random.default_rng(nmo)
    M = rng.standard_normal((nmo, naux, nmo))
    U = rng.standard_normal((naux, naux))
    t = bo.TCMatrix_gwbse(M.copy())
    threecenter.multiply_right_with_aux_matrix(t, U)
    ref = np.einsum("mpn,pq->mqn", M.astype(np.longdouble), U.astype(np.longdouble))
    bound = naux * 2.0**-53 * np.abs(M).max(axis=1)[:, None, :] * np.abs(U).max(axis=0)[None, :, None]
    assert np.all(np.abs(t.data - ref).astype(np.float64) <= bound + 2.0**-52 * np.abs(t.data))
