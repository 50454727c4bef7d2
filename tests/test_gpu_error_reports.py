"""A bounded wait of the tensor-core FP64 products that gives up leaves a code in a page-locked slot of
the workspace.  Every call that waits for its products must return it as BSE_ERR_TIMEOUT, and only
that call.  The code is planted from the host here; no wait runs out."""
import ctypes

import numpy as np
import pytest

import native
from votca_gb300 import _lib
from votca_gb300 import bse_operator as bo
from votca_gb300.davidson import DavidsonSolver
from votca_gb300.synthetic import Problem

pytestmark = pytest.mark.gpu

TIMEOUT = 4
P = lambda a: a.ctypes.data_as(_lib.c_dp)
I4 = ctypes.c_int32 * 4


def _context(seed=5, v=4, c=20, naux=30, precision=bo.PRECISION_FP64):
    p = Problem(v=v, c=c, naux=naux, nmo=v + c, seed=seed)
    opt = bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)
    return bo.GpuBSEContext(p.w, bo.TCMatrix_gwbse(p.mmn), p.hqp, opt, precision=precision)


def _plant(ctx, code=13):
    native.load().shim_plant_error(ctx.handle, code)


def _times_out(call):
    with pytest.raises(_lib.BSEError) as e:
        call()
    assert e.value.code == TIMEOUT


def _vectors(ctx, k, seed=1):
    return np.asfortranarray(np.random.default_rng(seed).standard_normal((ctx.size, k)))


@pytest.mark.parametrize("full", [False, True])
def test_gradient(full):
    ctx = _context()
    X, Y, g = _vectors(ctx, 2), 0.1 * _vectors(ctx, 2, 2), np.ones(2)
    gw = np.zeros(30)

    def call():
        if full:
            _lib.check(ctx._L.bse_op_eig_gradient_full(ctx.handle, I4(1, 2, 1, 0), I4(0, 2, 0, 1), P(X), P(Y), ctx.size,
                                                       2, P(g), None, None, P(gw)))
        else:
            _lib.check(ctx._L.bse_op_eig_gradient(ctx.handle, 1, 2, 1, 0, P(X), ctx.size, 2, P(g), None, None, P(gw)))

    call()
    _plant(ctx)
    _times_out(call)
    call()
    ctx.close()


def test_gradient_device():
    import torch

    ctx = _context()
    X = torch.from_numpy(_vectors(ctx, 2).T.copy()).cuda()
    gw = torch.zeros(30, dtype=torch.float64, device="cuda")
    g = np.ones(2)

    def call():
        _lib.check(ctx._L.bse_op_eig_gradient_device(ctx.handle, I4(1, 2, 1, 0), None, X.data_ptr(), None, ctx.size, 2,
                                                     P(g), None, None, None, None, None, gw.data_ptr(),
                                                     torch.cuda.current_stream().cuda_stream))

    call()
    _plant(ctx)
    _times_out(call)
    call()
    ctx.close()


@pytest.mark.parametrize("name", ["shim_stage_dense_screening", "shim_stage_dense_screening_uks"])
def test_dense_screening_staging(name):
    v, c, naux = 4, 20, 30
    p = Problem(v=v, c=c, naux=naux, nmo=v + c, seed=5)
    M = bo.TCMatrix_gwbse(p.mmn)
    d = _lib.bse_mmn_desc(M.auxsize(), M.get_mmin(), M.get_mmax(), M.get_nmin(), M.get_nmax())
    ptrs = (_lib.c_dp * M.msize())(*[ctypes.cast(M.data.ctypes.data + m * M.data.strides[0], _lib.c_dp)
                                     for m in range(M.msize())])
    W = np.asfortranarray(np.diag(p.w))
    h = np.asfortranarray(p.hqp)
    o = _lib.bse_options(v - 1, 0, 0, 0, v + c - 1)
    L = native.load()
    run = lambda code: getattr(L, name)(ctypes.byref(d), ptrs, P(W), P(h), ctypes.c_int64(h.shape[0]), ctypes.byref(o),
                                        code)
    assert run(0) == 0, L.shim_last_error()
    assert run(13) == TIMEOUT
    assert run(0) == 0


@pytest.mark.parametrize("which", [[0], [1], [2], [0, 1, 2]])
def test_lockstep_batch(which):
    """Every molecule's products, whichever place it has in the batch, and of several none is left over."""
    ctxs = [_context(seed=s, c=c) for s, c in ((5, 20), (6, 31), (7, 12))]
    ops = [bo.SingletOperator_TDA(x) for x in ctxs]

    def call():
        ds = DavidsonSolver()
        ds.set_tolerance(1e-7)
        return ds.solve_batch(ops, 2)

    ref = call()[0]
    for w in which:
        _plant(ctxs[w])
    _times_out(call)
    np.testing.assert_array_equal(call()[0], ref)
    for x in ctxs:
        x.close()


@pytest.mark.parametrize("which", ["dense", "factorised"])
def test_lockstep_batch_engines(which):
    """The grouped tensor-core products report into the first engine of their group, which need not be
    the first molecule's: an FP64 molecule first, then one without a dense form (off-diagonal Hqp)
    and one with it."""
    p = Problem(v=4, c=18, naux=30, nmo=22, seed=6)
    h = p.hqp.copy()
    h[5, 6] = h[6, 5] = 1e-3
    opt = bo.BSEOperator_Options(homo=3, rpamin=0, qpmin=0, vmin=0, cmax=21)
    ctxs = [_context(seed=5), bo.GpuBSEContext(p.w, bo.TCMatrix_gwbse(p.mmn), h, opt, precision=bo.PRECISION_MIXED),
            _context(seed=7, c=16, precision=bo.PRECISION_MIXED)]
    ops = [bo.SingletOperator_TDA(x) for x in ctxs]

    def call():
        ds = DavidsonSolver()
        ds.set_tolerance(1e-5)
        return ds.solve_batch(ops, 2)

    call()
    native.load().shim_plant_engine_error(ctxs[2 if which == "dense" else 1].handle, 3)
    _times_out(call)
    call()
    for x in ctxs:
        x.close()


def test_dense_forms_are_not_kept_after_an_error():
    """The dense forms of a batch are built on its first solve, with the smallest operator's engine."""
    ctxs = [_context(seed=5, c=24, precision=bo.PRECISION_MIXED), _context(seed=7, c=16, precision=bo.PRECISION_MIXED)]
    ops = [bo.SingletOperator_TDA(x) for x in ctxs]

    def call():
        ds = DavidsonSolver()
        ds.set_tolerance(1e-5)
        return ds.solve_batch(ops, 2)

    native.load().shim_plant_engine_error(ctxs[1].handle, 3)
    _times_out(call)
    evals, info, _ = call()
    assert all(i == "Success" for i in info)
    for x in ctxs:
        x.close()


@pytest.mark.parametrize("M,N,K", [(640, 64, 512), (2000, 130, 230), (300, 40, 4000)])
def test_wait_limit(M, N, K):
    """Waits that give up at once, with loads and MMAs in flight: an error, and the next product is right."""
    L = native.load()
    rng = np.random.default_rng(M)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    v = np.array([M, N, K, 1, 1, K, 1, 0, 0, N, 1, 0, 0, N, 1, 0, 0], dtype=np.int64)

    def run(us):
        C, taken, keep = np.zeros((M, N)), ctypes.c_int(), ctypes.c_int64()
        n = lambda a: ctypes.c_int64(a.size)
        rc = L.shim_oz_dgemm(P(v.view(np.float64)), P(A), n(A), P(B), n(B), P(C), n(C), ctypes.c_double(1.0),
                             ctypes.c_double(0.0), ctypes.c_int64(1 << 30), us, ctypes.byref(taken),
                             ctypes.byref(keep))
        assert taken.value == 1
        return rc, C

    assert run(0)[0] == TIMEOUT
    rc, C = run(2000000)
    assert rc == 0
    bound = K * 2.0**-53 * np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=0)[None, :]
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble)
    assert np.all(np.abs(C - ref) <= bound + 2.0**-52 * np.abs(ref))


def test_workspace_and_engine_at_once():
    """A split-precision handle with a code in its workspace and one in its engine: one call reports both."""
    ctx = _context(precision=bo.PRECISION_MIXED)
    op = bo.SingletOperator_TDA(ctx)
    X = _vectors(ctx, 3)
    ref = op.matmul(X)
    _plant(ctx)
    native.load().shim_plant_engine_error(ctx.handle, 3)
    _times_out(lambda: op.matmul(X))
    np.testing.assert_array_equal(op.matmul(X), ref)
    ctx.close()
