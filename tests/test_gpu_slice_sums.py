"""The sum over the K groups of a slice product: the partial sums (float pairs, exact here) must be added as
FP64 numbers.  Each group is one digit run with its own scale, so a large sum, a small one and the large
one's negative leave the small one, which is 27 bits below the low part of the large: 24-bit low words
lose it."""
import ctypes

import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu


# 3 to 23 runs of 1024, each a group of its own for a product this small
@pytest.mark.parametrize("runs", [3, 7, 12, 23])
@pytest.mark.parametrize("M,N", [(1, 1), (130, 33), (40, 70)])
def test_groups_are_added_in_fp64(M, N, runs):
    chain, L = 1024, native.load()
    A, B = np.zeros((M, runs * chain)), np.zeros((N, runs * chain))
    big = 1.0 + 2.0**-12  # big^2 = 1 + 2^-11 + 2^-24: the last term is the pair's low part
    A[:, 5], B[:, 5] = big, big
    A[:, chain + 9], B[:, chain + 9] = 2.0**-26, 2.0**-25
    A[:, (runs - 1) * chain + 1], B[:, (runs - 1) * chain + 1] = big, -big
    C = np.zeros((M, N), order="F")
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    i = ctypes.c_int64
    assert L.shim_slice_gemm(p(A), p(B), i(M), i(N), i(runs * chain), i(chain), p(C)) == 0, L.shim_last_error()
    assert np.all(C == 2.0**-51)
