"""Lockstep solves at the edges of their grouped kernels: molecules from one row tile to many row
chunks in one batch, new columns that fit the Gram-Schmidt kernel's shared memory and that do not
(n / 4 x columns x 8 bytes beyond 200 KB), and one to twelve roots (outputs of the transposed
products from less than a warp to several per thread).

Converged to a residual norm of 1e-7, an FP64 eigenvalue is off by at most the residual (and by
its square over the gap where that is larger than 1e-7): 1e-7 against the dense eigenvalues
bounds both, and 2e-7 the difference of two such solves.
"""
import numpy as np
import pytest

from votca_gb300.synthetic import Problem

pytestmark = pytest.mark.gpu


def _ops(shapes):
    from votca_gb300 import bse_operator as bo

    ctxs = []
    for v, c, naux, seed in shapes:
        p = Problem(v=v, c=c, naux=naux, nmo=v + c, seed=seed)
        opt = bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)
        ctxs.append(bo.GpuBSEContext(p.w, bo.TCMatrix_gwbse(p.mmn), p.hqp, opt, precision=bo.PRECISION_FP64))
    return ctxs, [bo.SingletOperator_TDA(ctx) for ctx in ctxs]


def _solver():
    from votca_gb300.davidson import DavidsonSolver

    ds = DavidsonSolver()
    ds.set_tolerance(1e-7)
    return ds


@pytest.mark.parametrize("roots,shapes", [
    (1, [(3, 10, 12, 1), (2, 16, 8, 2), (8, 65, 24, 3)]),
    (5, [(2, 15, 8, 4), (7, 73, 20, 5), (16, 64, 16, 6), (9, 57, 16, 7)]),   # n = 30, 511, 1024, 513
    (12, [(4, 32, 24, 8), (5, 103, 16, 9), (3, 171, 12, 10)]),
])
def test_lockstep_sizes(roots, shapes):
    ctxs, ops = _ops(shapes)
    ev, info, _ = _solver().solve_batch(ops, roots)
    assert all(i == "Success" for i in info)
    for m, op in enumerate(ops):
        H = op.matmul(np.eye(op.rows()))
        np.testing.assert_allclose(ev[m], np.linalg.eigvalsh(0.5 * (H + H.T))[:roots], rtol=0, atol=1e-7)
    for ctx in ctxs:
        ctx.close()


def test_lockstep_large_beside_small():
    """n = 15360 with 5 roots (new columns beyond the shared memory of a CTA) beside n = 30."""
    ctxs, ops = _ops([(60, 256, 12, 11), (2, 15, 8, 12)])
    ev, info, _ = _solver().solve_batch(ops, 5)
    assert all(i == "Success" for i in info)
    for m, op in enumerate(ops):
        lam, _ = _solver().solve(op, 5)
        np.testing.assert_allclose(ev[m], lam, rtol=0, atol=2e-7)
    for ctx in ctxs:
        ctx.close()
