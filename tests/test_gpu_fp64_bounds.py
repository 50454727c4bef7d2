"""What an FP64 product promises (include/votca_gb300_bse.h, BSE_PRECISION_FP64): an element of a contraction
A X of K terms is off by at most K 2^-53 max|row of A| max|column of X|, whatever path its size takes; by at
most K 2^-53 sum |a||x| where A and X are graded in opposite directions along K, by more than 12 bits; and
bse_op_matmul_device_noalloc, which runs FMA chains throughout, always by that.

The inputs are those where the two differ: opposed gradings, and a large element of X against zeros of
A.  The largest error in units of K 2^-53 sum |a||x| is printed."""
import ctypes

import numpy as np
import pytest

from votca_gb300 import _lib
from votca_gb300 import bse_operator as bo
from votca_gb300.synthetic import Problem

pytestmark = pytest.mark.gpu

U = 2.0**-53


def _operands(kind, n, k, rng):
    A, X = rng.standard_normal((n, n)), rng.standard_normal((n, k))
    if kind.startswith("opposed"):
        d = 10.0 ** np.linspace(0, float(kind[7:]), n)
        return A / d[None, :], X * d[:, None]
    if kind == "one_large":  # one element of every vector, zero in half of the rows that meet it
        X *= 1e-12
        j = rng.integers(0, n, k)
        X[j, np.arange(k)] = 1.0
        A[np.ix_(np.arange(0, n, 2), np.unique(j))] = 0.0
    return A, X


@pytest.mark.parametrize("kind", ["gauss", "opposed3", "opposed6", "opposed10", "opposed20", "opposed80", "one_large"])
@pytest.mark.parametrize("n,k", [(129, 17), (700, 70), (1300, 33)])  # FMA chains; digit products; two runs
@pytest.mark.parametrize("scaled", [False, True])
def test_bounds(kind, n, k, scaled):
    rng = np.random.default_rng(n)
    A, X = _operands(kind, n, k, rng)
    if scaled:  # rows and columns of different scales, and some that are zero
        A *= 2.0 ** rng.integers(-60, 60, (n, 1))
        X *= 2.0 ** rng.integers(-60, 60, (1, k))
        A[3] = 0.0
        X[:, 2] = 0.0
    op = bo.DenseGpuOperator(A)
    Y = op.matmul(X)
    op.close()
    err = np.abs(Y - A.astype(np.longdouble) @ X.astype(np.longdouble)).astype(np.float64)
    largest = np.abs(A).max(axis=1)[:, None] * np.abs(X).max(axis=0)[None, :]
    terms = np.abs(A) @ np.abs(X)
    opposed = kind.startswith("opposed") and float(kind[7:]) > 5  # of 10; Gaussian factors bring elements closer
    assert np.all(err <= n * U * (terms if opposed else largest) + 2.0**-52 * np.abs(Y))
    print(kind, n, k, float((err[terms > 0] / (n * U * terms[terms > 0])).max()))


@pytest.mark.parametrize("kind", ["gauss", "graded", "one_large"])
def test_noalloc_keeps_the_bound_of_the_terms(kind):
    import torch

    v, c, naux, k = 8, 64, 256, 6
    rng = np.random.default_rng(9)
    p = Problem(v=v, c=c, naux=naux, nmo=v + c, seed=9)
    opt = bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)
    ctx = bo.GpuBSEContext(p.w, bo.TCMatrix_gwbse(p.mmn), p.hqp, opt)
    X = rng.standard_normal((v * c, k))
    if kind == "graded":
        X *= 10.0 ** rng.uniform(-15, 0, X.shape)
    if kind == "one_large":
        X *= 1e-12
        X[rng.integers(0, v * c, k), np.arange(k)] = 1.0
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    dY = torch.zeros_like(dX)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(ctx._L.bse_op_matmul_device_noalloc(ctx.handle, 0, 1, 0, 0, ctypes.c_void_p(dX.data_ptr()), v * c, k,
                                                   ctypes.c_void_p(dY.data_ptr()), v * c, stream))
    torch.cuda.synchronize()
    ctx.close()
    B = np.ascontiguousarray(p.mmn[:v, :, v:].transpose(0, 2, 1)).reshape(v * c, naux)
    Bl = B.astype(np.longdouble)
    err = np.abs(dY.cpu().numpy().T - Bl @ (Bl.T @ X.astype(np.longdouble))).astype(np.float64)
    terms = np.abs(B) @ (np.abs(B).T @ np.abs(X))
    assert np.all(err <= 1.01 * (v * c + naux) * U * terms)
