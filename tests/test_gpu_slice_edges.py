"""Slice products (BSE_PRECISION_SLICED) at the edges of their kernels, against the FP64 path.

The digit planes are cut per run of K elements (the largest multiple of 64 up to 1024 that divides
the padded K), the level sums leave the tensor core every 512 of them, tiles are 128 x 64 or
128 x 32, and the runs of a tile may go to several CTAs: the shapes below end in every run length
class of the slicer, in whole, short and single drain intervals, and on both sides of the tiles.

Tolerance: five digits of 7 bits keep every operand to 2^-36 of its run's largest element, and the
dropped digit levels are 2^-35 of the two scales; for Gaussian data, whose largest element is three to
four times the typical one, that is up to 16 x 2^-35 x sqrt(2) = 7e-10 of a product term in each
of the (at most) two stages with independent signs, far less in a sum of K terms: 3e-10 of the
product norm, as for the other slice products.
"""
import numpy as np
import pytest

import oracle
from votca_gb300.synthetic import Problem

pytestmark = pytest.mark.gpu

SLICED_TOL = 3e-10


def contexts(p, v, c):
    from votca_gb300 import bse_operator as bo

    Mmn = bo.TCMatrix_gwbse(p.mmn)
    opt = bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)
    return [bo.GpuBSEContext(p.w, Mmn, p.hqp, opt, precision=q) for q in (bo.PRECISION_FP64, bo.PRECISION_SLICED)]


@pytest.mark.parametrize("v,c,naux,k", [
    (1, 31, 64, 127),    # stage 2: one run of 64; 127 vectors
    (2, 33, 64, 64),     # run of 128; 128 rows of X
    (3, 63, 64, 43),     # run of 192; 129 rows
    (4, 64, 80, 3),      # run of 320
    (4, 65, 112, 2),     # run of 448
    (4, 40, 144, 9),     # run of 576: a drain interval and one stage pair
    (4, 40, 176, 1),     # run of 704
    (4, 40, 208, 5),     # run of 832
    (32, 20, 32, 4),     # run of 1024, N = 32
    (33, 20, 64, 4),     # N = 33; 2112 = 3 runs of 704
    (64, 12, 17, 2),     # N = 64; 1088: 17 runs of 64, shared by several CTAs
    (65, 12, 33, 2),     # two column blocks
    (2, 1088, 24, 3),    # stage 1 and the exchange in runs of 64
])
def test_slice_edges(v, c, naux, k):
    from votca_gb300 import bse_operator as bo

    f, s = contexts(Problem(v=v, c=c, naux=naux, nmo=v + c, seed=61), v, c)
    X = np.random.default_rng(61).standard_normal((v * c, k))
    for op in ("hx", "hd", "hd2"):
        yf = bo.BSE_OPERATOR(f, *oracle.OPERATORS[op]).matmul(X)
        ys = bo.BSE_OPERATOR(s, *oracle.OPERATORS[op]).matmul(X)
        assert np.linalg.norm(ys - yf) < SLICED_TOL * np.linalg.norm(yf), op


def test_slice_scales_and_zeros():
    """Vectors of very different norms and a zero vector in one product: each keeps its own scale."""
    from votca_gb300 import bse_operator as bo

    v, c, naux = 6, 50, 96
    f, s = contexts(Problem(v=v, c=c, naux=naux, nmo=v + c, seed=62), v, c)
    X = np.random.default_rng(62).standard_normal((v * c, 5)) * np.array([1e-25, 1.0, 0.0, 1e25, 1e-3])
    for op in ("hx", "hd", "hd2"):
        yf = bo.BSE_OPERATOR(f, *oracle.OPERATORS[op]).matmul(X)
        ys = bo.BSE_OPERATOR(s, *oracle.OPERATORS[op]).matmul(X)
        assert not ys[:, 2].any()
        err, ref = np.linalg.norm(ys - yf, axis=0), np.linalg.norm(yf, axis=0)
        assert (err <= SLICED_TOL * ref).all(), (op, err / np.maximum(ref, 1e-300))
