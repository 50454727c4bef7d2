"""FP64 Davidson solves whose blocks of new columns have one to more than 64 members: the block
orthonormalisation runs as Cholesky QR up to 64 columns and column by column beyond, and the small
eigenproblem without divisions in its reflectors.

Converged to a residual norm of 1e-7, an eigenvalue is off by at most the residual: 1e-7 against the
dense eigenvalues.  The Ritz vectors of a Rayleigh-Ritz projection onto an orthonormal basis are
orthonormal as far as the basis and the small eigenvectors are: n eps each, 1e-11 with room for the
reorthogonalisation's constant.
"""
import numpy as np
import pytest

from votca_gb300.synthetic import Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("roots", [1, 2, 3, 11, 16, 22, 32, 43, 60])
def test_block_sizes(roots):
    from votca_gb300 import bse_operator as bo
    from votca_gb300.davidson import DavidsonSolver

    v, c, naux = 9, 61, 24
    p = Problem(v=v, c=c, naux=naux, nmo=v + c, seed=71)
    opt = bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)
    ctx = bo.GpuBSEContext(p.w, bo.TCMatrix_gwbse(p.mmn), p.hqp, opt, precision=bo.PRECISION_FP64)
    op = bo.SingletOperator_TDA(ctx)
    ds = DavidsonSolver()
    ds.set_tolerance(1e-7)
    ds.set_max_search_space(max(50, 6 * roots))
    lam, X = ds.solve(op, roots)
    H = op.matmul(np.eye(v * c))
    np.testing.assert_allclose(lam, np.linalg.eigvalsh(0.5 * (H + H.T))[:roots], rtol=0, atol=1e-7)
    X = np.asarray(X)
    assert np.abs(X.T @ X - np.eye(roots)).max() < 1e-11
    ctx.close()
