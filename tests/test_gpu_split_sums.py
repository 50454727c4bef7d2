"""The sum over the K splits of split-precision products where the splits' magnitudes lie close
together (integer sums), far apart (FP64 sums) or are zero.

The products are accurate to 5e-5 of the interaction part whatever the splits' sums are made of:
three bf16 products (2^-16 per term) and FP32 chains, with the splits added exactly or in FP64.
"""
import numpy as np
import pytest

import oracle
from votca_gb300.synthetic import Problem

pytestmark = pytest.mark.gpu

MIXED_TOL = 5e-5


@pytest.mark.parametrize("decades", [0, 3, 8, 14])
@pytest.mark.parametrize("zero_half", [False, True])
def test_split_sums(decades, zero_half):
    from votca_gb300 import bse_operator as bo

    v, c, naux, k = 8, 70, 320, 5
    p = Problem(v=v, c=c, naux=naux, nmo=v + c, seed=81)
    scale = 10.0 ** (-decades * np.arange(naux) / naux)  # K = (P, v): a split is a range of P
    if zero_half:
        scale[naux // 2:] = 0.0
    mmn = p.mmn * scale[None, :, None]
    opt = bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)
    f, m = [bo.GpuBSEContext(p.w, bo.TCMatrix_gwbse(mmn), p.hqp, opt, precision=q)
            for q in (bo.PRECISION_FP64, bo.PRECISION_MIXED)]
    X = np.random.default_rng(81).standard_normal((v * c, k))
    for op in ("hx", "hd", "hd2"):
        yf = bo.BSE_OPERATOR(f, *oracle.OPERATORS[op]).matmul(X)
        ym = bo.BSE_OPERATOR(m, *oracle.OPERATORS[op]).matmul(X)
        assert np.linalg.norm(ym - yf) < MIXED_TOL * np.linalg.norm(yf), op
    f.close()
    m.close()
