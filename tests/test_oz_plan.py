"""CPU test of the plan behind the tensor-core FP64 GEMM (votca_gb300/csrc/oz_plan.hpp): for every
operand order, batch form, odd size, K split and chunk it must write each output once, with the
sum that the strided loops give."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("oz") / "oz_plan_shim.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "oz_plan_shim.cpp"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


# which operands a batch moves: "a", "b", "ab" or "" (none)
@pytest.mark.parametrize("m1,m2", list(itertools.product(["-", "a", "b", "ab"], ["-", "a", "b", "ab"])))
@pytest.mark.parametrize("at,bt,ct", [(0, 0, 0), (1, 0, 0), (0, 1, 1), (1, 1, 1)])
def test_plan_covers_every_output_once(lib, m1, m2, at, bt, ct):
    rng = np.random.default_rng(17)
    for M, N, K, sms, budget in ((5, 3, 7, 4, 1 << 40), (130, 65, 300, 8, 1 << 40), (300, 9, 40, 2, 60000),
                                 (9, 300, 513, 152, 1 << 40), (1, 70, 33, 3, 1 << 14)):
        n1, n2 = (1 if m1 == "-" else 3), (1 if m2 == "-" else 2)
        if M * N * K * n1 * n2 > 6_000_000:
            K = 35
        ab = [M * K if "a" in m else 0 for m in (m1, m2)]
        bb = [K * N if "b" in m else 0 for m in (m1, m2)]
        if ab[0] and ab[1]:
            ab[0] *= n2
        if bb[0] and bb[1]:
            bb[0] *= n2
        A = rng.integers(-4, 5, M * K * n1 * n2).astype(np.float64)
        B = rng.integers(-4, 5, K * N * n1 * n2).astype(np.float64)
        C = rng.integers(-4, 5, M * N * n1 * n2).astype(np.float64)
        C2, counts = C.copy(), np.zeros(C.size, dtype=np.int32)
        v = [M, N, K, n1, n2] + ([K, 1] if at else [1, M]) + ab + ([N, 1] if bt else [1, K]) + bb
        v += ([N, 1] if ct else [1, M]) + [M * N * n2, M * N]
        v = np.array(v, dtype=np.int64)
        out = np.zeros(9, dtype=np.int64)
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        ok = lib.oz_plan_run(p(v), p(A), p(B), p(C), p(C2), ctypes.c_double(-2.0), ctypes.c_double(1.0),
                             ctypes.c_int64(sms), ctypes.c_int64(budget), p(counts), p(out))
        if not ok:  # only a plane budget below one tile refuses these forms
            assert budget < 1 << 20
            continue
        assert np.all(counts == 1)
        np.testing.assert_array_equal(C, C2)
        splits, kb_per, nkb = out[0], out[6], out[7]
        assert splits * kb_per >= nkb and (splits - 1) * kb_per < nkb
        assert splits == 1 or kb_per % 8 == 0


def test_plan_keeps_small_products_on_fma(lib):
    for M, N, K, want in ((64, 64, 64, 0), (200, 200, 3, 0), (16, 16, 512, 0)):
        v = np.array([M, N, K, 1, 1, 1, M, 0, 0, 1, K, 0, 0, 1, M, 0, 0], dtype=np.int64)
        out = np.zeros(9, dtype=np.int64)
        A, B, C = np.zeros(M * K), np.zeros(K * N), np.zeros(M * N)
        counts = np.zeros(M * N, dtype=np.int32)
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        assert lib.oz_plan_run(p(v), p(A), p(B), p(C), p(C.copy()), ctypes.c_double(1.0), ctypes.c_double(0.0),
                               ctypes.c_int64(152), ctypes.c_int64(1 << 30), p(counts), p(out))
        assert out[8] == want


@pytest.mark.parametrize("M,N,K,nb", [(1, 1, 1, 1), (60, 15, 8192, 1), (8192, 15, 60, 1), (64, 64, 64, 1),
                                      (65, 17, 300, 7), (900, 900, 64, 1), (30, 30, 100000, 2)])
def test_fma_plan(lib, M, N, K, nb):
    """Every K element is in one split; a fixed split keeps the chain the 64 x 64 tiles had."""
    v = np.array([M, N, K, nb], dtype=np.int64)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    for splitk in (0, -1, 1, 5):
        out = np.zeros(5, dtype=np.int64)
        lib.fma_plan_of(p(v), ctypes.c_int64(152), ctypes.c_int32(splitk), p(out))
        tm, tn, splits, kc, rule = (int(x) for x in out)
        assert tm in (16, 32, 64) and tn in (16, 32, 64) and tn <= tm
        assert kc % 16 == 0 and (splits - 1) * kc < K <= splits * kc
        if splitk != 0:
            want = rule if splitk < 0 else splitk
            chunk = -(-(-(-K // want)) // 16) * 16
            assert kc == chunk and splits == -(-K // chunk)
