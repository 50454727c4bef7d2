"""Performance cases of the GW-BSE exciton path: what a user's program asks of this library.

Every case is one pass through the public entry points (the Python mirror of VOTCA-XTP's
interface, which marshals into the C ABI).  The sizes are those of the benchmark (one small
molecule, a v64 c512 molecule, the batched molecules with v 4..32, c 32..256, Naux 128..1024)
and generic sizes between them, ragged ones included; the values follow
votca_gb300/synthetic.py.  Sizes: v occupied and c virtual levels of the BSE window, naux
auxiliary functions, k vectors of a product, roots of a solve.

  product    BSE_OPERATOR.matmul / matmul_device: cqp Hqp + cx Hx - cd Hd on k vectors
  ham        HamiltonianOperator.matmul: [[A, B], [-B, -A]] on k vectors (full BSE)
  solve      DavidsonSolver.solve of the TDA problem (solve_hermitian)
  full_solve Solve_nonhermitian_Davidson: full-BSE roots, X and Y
  batch      DavidsonSolver.solve_batch: many small molecules in lockstep
  gradient   eigenvalues and their gradients (staging, solve, Hellmann-Feynman backward)
  screening  RPA dielectric matrix and its inverse
  fill       three-centre integrals to MO basis, then the auxiliary metric
"""
import math

import numpy as np
import torch

from votca_gb300 import adjoint, bse, screening, threecenter
from votca_gb300 import bse_operator as bo
from votca_gb300.davidson import DavidsonSolver
from votca_gb300.synthetic import mmn_tensor_torch, qp_energies, screening_w

PRECISION = {"fp64": bo.PRECISION_FP64, "mixed": bo.PRECISION_MIXED, "sliced": bo.PRECISION_SLICED}
OPERATOR = {"singlet": bo.SingletOperator_TDA, "triplet": bo.TripletOperator_TDA}
COEF = {"singlet": (1.0, 2.0, 1.0), "triplet": (1.0, 0.0, 1.0)}  # cqp, cx, cd


def listed():
    return [
        # One product of the smallest benchmark molecule from host arrays: a caller that drives its
        # own eigensolver on a small molecule, where launches and copies count.
        dict(name="product_fp64_small", kind="product", precision="fp64", spin="singlet", v=8, c=64, naux=256, k=15,
             host=True),
        # The plain FP64 product (the default precision) of a medium molecule with ragged sizes, on
        # device vectors: the inner call of an FP64 Davidson solve.
        dict(name="product_fp64", kind="product", precision="fp64", spin="singlet", v=30, c=220, naux=900, k=15,
             host=False),
        # The headline product: split-precision singlet product of the v64 c512 molecule, 30 vectors
        # (one Davidson iteration of 20 roots).
        dict(name="product_mixed_large", kind="product", precision="mixed", spin="singlet", v=64, c=512, naux=2048,
             k=30, host=False),
        # FP64-accurate slice products of a larger molecule, 20 Ritz vectors: the polish of a
        # split-precision solve, and whole solves at this precision.
        dict(name="product_sliced", kind="product", precision="sliced", spin="singlet", v=32, c=256, naux=1024, k=20,
             host=False),
        # The full-BSE Hamiltonian on 10 vectors from host arrays (both blocks, Hd2 among them).
        dict(name="ham_mixed", kind="ham", precision="mixed", v=32, c=256, naux=1024, k=10),
        # Ten singlets of the smallest benchmark molecule in FP64: latency, small eigenproblems,
        # Gram-Schmidt.
        dict(name="solve_fp64_small", kind="solve", precision="fp64", spin="singlet", v=8, c=64, naux=256, roots=10),
        # Ten singlets of a larger molecule, split precision with the FP64-accurate polish.
        dict(name="solve_mixed", kind="solve", precision="mixed", spin="singlet", v=32, c=256, naux=1024, roots=10),
        # Five full-BSE roots of a medium molecule at the default precision.
        dict(name="full_solve_fp64", kind="full_solve", precision="fp64", v=16, c=100, naux=400, roots=5),
        # A screening campaign over many small molecules: five singlets of each, in lockstep.
        dict(name="batch_mixed", kind="batch", precision="mixed", spin="singlet", molecules=24, roots=5),
        # Eigenvalues and their gradients with respect to Mmn, Hqp and the screening: one step of a
        # geometry optimisation or a fit, forward and backward.
        dict(name="gradient_fp64", kind="gradient", precision="fp64", v=12, c=90, naux=300, roots=3),
        # The dielectric matrix of a molecule and its inverse: once per GW-BSE run, and once per
        # frequency of the perturbative dynamical screening.
        dict(name="screening_fp64", kind="screening", v=32, c=256, naux=1000),
        # The Mmn tensor from AO integrals: AO to MO transform and the auxiliary metric.
        dict(name="fill_fp64", kind="fill", nbf=210, nmo=160, naux=500),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "product", "ham", "solve", "solve", "full_solve", "batch",
                       "gradient", "screening", "fill"])
    v, c, naux = rng.randint(4, 32), _log_int(rng, 32, 256), _log_int(rng, 128, 1024)
    if kind == "product":
        precision = rng.choice(["fp64", "mixed", "sliced"])
        if precision != "fp64" and rng.random() < 0.4:
            v, c, naux = rng.randint(24, 56), rng.randint(200, 440), rng.randint(600, 1500)
        return dict(kind="product", precision=precision, spin=rng.choice(["singlet", "triplet"]), v=v, c=c, naux=naux,
                    k=_log_int(rng, 2, 40), host=rng.random() < 0.25)
    if kind == "ham":
        return dict(kind="ham", precision=rng.choice(["fp64", "mixed", "sliced"]), v=v, c=min(c, 200),
                    naux=min(naux, 700), k=rng.randint(2, 16))
    if kind == "solve":
        return dict(kind="solve", precision=rng.choice(["fp64", "mixed", "sliced"]),
                    spin=rng.choice(["singlet", "triplet"]), v=rng.randint(4, 24), c=_log_int(rng, 32, 160),
                    naux=_log_int(rng, 128, 600), roots=rng.randint(3, 10))
    if kind == "full_solve":
        return dict(kind="full_solve", precision=rng.choice(["fp64", "mixed"]), v=rng.randint(6, 16),
                    c=_log_int(rng, 32, 110), naux=_log_int(rng, 128, 420), roots=rng.randint(2, 5))
    if kind == "batch":
        return dict(kind="batch", precision="mixed", spin=rng.choice(["singlet", "triplet"]),
                    molecules=rng.randint(4, 24), roots=rng.randint(3, 6))
    if kind == "gradient":
        return dict(kind="gradient", precision="fp64", v=rng.randint(4, 12), c=_log_int(rng, 32, 96),
                    naux=_log_int(rng, 128, 320), roots=rng.randint(1, 4))
    if kind == "screening":
        return dict(kind="screening", v=v, c=c, naux=naux)
    nbf = rng.randint(60, 220)
    return dict(kind="fill", nbf=nbf, nmo=rng.randint(nbf // 2, nbf), naux=_log_int(rng, 128, 520))


# ---- inputs ----


def _molecule(seed, v, c, naux, nmo=None):
    """Mmn (m, P, n), the diagonal Hqp and the diagonal screening of one synthetic molecule."""
    mmn = mmn_tensor_torch(seed, naux, nmo if nmo is not None else v + c)
    return mmn, np.diag(qp_energies(seed, v, c)), screening_w(seed, naux)


def _window(v, c):
    return bo.BSEOperator_Options(homo=v - 1, rpamin=0, qpmin=0, vmin=0, cmax=v + c - 1)


def _context(seed, case):
    mmn, hqp, w = _molecule(seed, case["v"], case["c"], case["naux"])
    return bo.GpuBSEContext(w, bo.TCMatrix_gwbse(mmn), hqp, _window(case["v"], case["c"]),
                            precision=PRECISION[case["precision"]])


def _vectors(seed, rows, k):
    """k normalised trial vectors, one per row."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    X = torch.randn((k, rows), generator=g, dtype=torch.float64, device="cuda")
    return X / X.norm(dim=1, keepdim=True)


def _batch_shapes(case, seed):
    """Molecules of the batched benchmark's ranges; the shapes belong to the case, the values to the seed."""
    rs = np.random.RandomState(1000 + 31 * case["molecules"] + case["roots"])
    n = case["molecules"]
    vs, cs, ps = rs.randint(4, 33, n), rs.randint(32, 257, n), rs.randint(128, 1025, n)
    return [(int(vs[i]), int(cs[i]), int(ps[i]), seed * 131 + i) for i in range(n)]


def _ao_inputs(seed, nbf, nmo, naux):
    g = torch.Generator(device="cuda").manual_seed(seed + 5)
    kw = dict(generator=g, dtype=torch.float64, device="cuda")
    ao = torch.randn((naux, nbf, nbf), **kw) / math.sqrt(nbf)
    C = torch.linalg.qr(torch.randn((nbf, nbf), **kw))[0][:, :nmo]
    U = torch.eye(naux, dtype=torch.float64, device="cuda") + torch.randn((naux, naux), **kw) * (0.3 / math.sqrt(naux))
    return 0.5 * (ao + ao.transpose(1, 2)), C, U


def prepare(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "product":
        ctx = _context(seed, case)
        X = _vectors(seed, ctx.size, case["k"])
        op = OPERATOR[case["spin"]](ctx)
        if case["host"]:
            return dict(kind=kind, op=op, X=np.asfortranarray(X.cpu().numpy().T), host=True)
        return dict(kind=kind, op=op, X=X, Y=torch.empty_like(X), host=False)
    if kind == "ham":
        ctx = _context(seed, case)
        X = _vectors(seed, 2 * ctx.size, case["k"])
        return dict(kind=kind, op=bo.HamiltonianOperator(bo.SingletOperator_TDA(ctx), bo.SingletOperator_BTDA_B(ctx)),
                    X=np.asfortranarray(X.cpu().numpy().T))
    if kind == "solve":
        return dict(kind=kind, op=OPERATOR[case["spin"]](_context(seed, case)), roots=case["roots"])
    if kind == "full_solve":
        ctx = _context(seed, case)
        return dict(kind=kind, A=bo.SingletOperator_TDA(ctx), B=bo.SingletOperator_BTDA_B(ctx), roots=case["roots"])
    if kind == "batch":
        ops = []
        for v, c, naux, sd in _batch_shapes(case, seed):
            ops.append(OPERATOR[case["spin"]](_context(sd, dict(case, v=v, c=c, naux=naux))))
        return dict(kind=kind, ops=ops, roots=case["roots"])
    if kind == "gradient":
        mmn, hqp, w = _molecule(seed, case["v"], case["c"], case["naux"])
        t = [torch.from_numpy(np.ascontiguousarray(a)).requires_grad_(True) for a in (mmn, hqp, w)]
        g = torch.linspace(1.0, 2.0, case["roots"], dtype=torch.float64)
        return dict(kind=kind, t=t, g=g, opt=_window(case["v"], case["c"]), roots=case["roots"],
                    precision=PRECISION[case["precision"]])
    if kind == "screening":
        v, c = case["v"], case["c"]
        mmn, hqp, _ = _molecule(seed, v, c, case["naux"])
        return dict(kind=kind, mmn=bo.TCMatrix_gwbse(mmn), e=np.diag(hqp).copy(), window=(v - 1, 0, v + c - 1))
    ao, C, U = _ao_inputs(seed, case["nbf"], case["nmo"], case["naux"])
    return dict(kind=kind, ao=ao.cpu().numpy(), C=np.asfortranarray(C.cpu().numpy()),
                U=np.asfortranarray(U.cpu().numpy()),
                mmn=bo.TCMatrix_gwbse.Initialize(case["naux"], 0, case["nmo"] - 1, 0, case["nmo"] - 1))


def run(s):
    kind = s["kind"]
    if kind == "product":
        if s["host"]:
            return s["op"].matmul(s["X"])
        X, Y = s["X"], s["Y"]
        s["op"].matmul_device(X.data_ptr(), X.shape[1], X.shape[0], Y.data_ptr(), Y.shape[1],
                              torch.cuda.current_stream().cuda_stream)
        return Y
    if kind == "ham":
        return s["op"].matmul(s["X"])
    if kind == "solve":
        opt = bse.DavidsonOptions(davidson_tolerance=1e-7, nmax=s["roots"])
        evals, evecs, ds = bse.solve_hermitian(s["op"], opt)
        return dict(evals=evals, evecs=evecs, success=ds.info() == "Success")
    if kind == "full_solve":
        opt = bse.DavidsonOptions(davidson_tolerance=1e-7, nmax=s["roots"])
        evals, X, Y, ds = bse.solve_nonhermitian_davidson(s["A"], s["B"], opt)
        return dict(evals=evals, X=X, Y=Y, success=ds.info() == "Success")
    if kind == "batch":
        ds = DavidsonSolver()
        ds.set_tolerance(1e-5)
        evals, info, _ = ds.solve_batch(s["ops"], s["roots"])
        return dict(evals=evals, success=[i == "Success" for i in info])
    if kind == "gradient":
        for x in s["t"]:
            x.grad = None
        lam = adjoint.bse_eigenvalues(*s["t"], s["opt"], s["roots"], precision=s["precision"])
        lam.backward(s["g"])
        return dict(evals=lam.detach(), mmn=s["t"][0].grad, hqp=s["t"][1].grad, w=s["t"][2].grad)
    if kind == "screening":
        eps = screening.rpa_epsilon(s["mmn"], s["e"], *s["window"])
        return dict(eps=eps, W=screening.cholesky_inverse(eps))
    threecenter.fill_3c_mo(s["mmn"], s["ao"], s["C"])
    threecenter.multiply_right_with_aux_matrix(s["mmn"], s["U"])
    return s["mmn"].data


# ---- what a pass cannot do without ----


def _product_work(v, c, naux, k, singlet, width):
    """Bytes and operations of k TDA columns: the cc and vv blocks (and the vc block of a singlet)
    at `width` bytes an element, the vectors in FP64."""
    vc = v * c
    flops = k * (2.0 * naux * vc * (v + c) + (4.0 * naux * vc if singlet else 0.0) + 2.0 * vc)
    return width * naux * (c * c + v * v + (vc if singlet else 0)) + 16.0 * vc * k, flops


def work(case):
    kind = case["kind"]
    width = 4.0 if case.get("precision") == "mixed" else 8.0
    singlet = case.get("spin", "singlet") == "singlet"
    if kind in ("product", "solve", "gradient"):
        # a solve cannot do without its first guess (2 roots columns) and two blocks of corrections
        k = case.get("k", 5 * case.get("roots", 0))
        b, f = _product_work(case["v"], case["c"], case["naux"], k, singlet, width)
        if kind == "gradient":  # the tensor is read and its gradient written
            n = case["v"] + case["c"]
            r, vc = case["roots"], case["v"] * case["c"]
            b += 16.0 * n * n * case["naux"]
            f += r * (4.0 * case["naux"] * vc * (case["v"] + case["c"]) + 4.0 * case["naux"] * vc)
        return dict(bytes=b, flops=f)
    if kind in ("ham", "full_solve"):
        # A and B on both halves of every vector; a full-BSE iteration applies the operator twice
        v, c, naux = case["v"], case["c"], case["naux"]
        k = 2 * case.get("k", 2 * 5 * case.get("roots", 0))
        b, f = _product_work(v, c, naux, k, True, width)
        return dict(bytes=b + width * naux * v * c, flops=f + k * naux * v * c * (4.0 * v + 4.0))
    if kind == "batch":
        b = f = 0.0
        for v, c, naux, _ in _batch_shapes(case, 0):
            pb, pf = _product_work(v, c, naux, 4 * case["roots"], singlet, width)
            b, f = b + pb, f + pf
        return dict(bytes=b, flops=f)
    naux = case["naux"]
    if kind == "screening":  # a symmetric rank update, and the inverse of a symmetric matrix
        vc = case["v"] * case["c"]
        return dict(bytes=8.0 * naux * vc + 16.0 * naux * naux, flops=1.0 * vc * naux * naux + 1.0 * naux**3)
    nbf, nmo = case["nbf"], case["nmo"]
    return dict(bytes=8.0 * naux * (nbf * nbf + nmo * nmo),
                flops=2.0 * naux * nbf * nmo * (nbf + nmo) + 2.0 * nmo * nmo * naux * naux)


# ---- the same in 64 bits with plain torch ----


def _blocks(seed, case):
    v, c, naux = case["v"], case["c"], case["naux"]
    mmn, hqp, w = _molecule(seed, v, c, naux)
    M = torch.from_numpy(mmn).cuda()  # (m, P, n)
    return M, torch.from_numpy(np.diag(hqp).copy()).cuda(), torch.from_numpy(w).cuda()


def _apply_exact(M, e, w, v, X, cqp, cx, cd, cd2=0.0):
    """(cqp Hqp + cx Hx - cd Hd - cd2 Hd2) on the rows of X (k, v * c)."""
    c = e.numel() - v
    naux, k = M.shape[1], X.shape[0]
    X3 = X.reshape(k, v, c)
    Y = cqp * (e[v:][None, None, :] - e[:v][None, :, None]) * X3
    vc = M[:v, :, v:]  # (v, P, c) = M(v, c, P)
    for P0 in range(0, naux, 64):
        Ps = slice(P0, min(naux, P0 + 64))
        if cx:
            b = vc[:, Ps, :].permute(1, 0, 2).reshape(-1, v * c)
            Y = Y + cx * ((X @ b.T) @ b).reshape(k, v, c)
        n = Ps.stop - P0
        if cd:  # Y[j, v1, c1] -= cd sum_P w_P M(v1, v, P) M(c1, c, P) X[j, v, c]
            cc = M[v:, Ps, v:].permute(1, 0, 2).reshape(n * c, c)  # rows (P, c1)
            S = (X3.reshape(k * v, c) @ cc.T).reshape(k, v, n, c)  # (j, v, P, c1)
            g = (M[:v, Ps, :v] * w[Ps][None, :, None]).permute(0, 2, 1).reshape(v, v * n)  # v1, (v, P)
            Y = Y - cd * torch.matmul(g, S.reshape(k, v * n, c))
        if cd2:  # Y[j, v1, c1] -= cd2 sum_P w_P M(c1, v, P) M(v1, c, P) X[j, v, c]
            b = vc[:, Ps, :].permute(1, 0, 2).reshape(n * v, c)  # rows (P, v1)
            U = (X3.reshape(k * v, c) @ b.T).reshape(k, v, n, v)  # (j, v, P, v1)
            a = (M[v:, Ps, :v] * w[Ps][None, :, None]).permute(0, 2, 1).reshape(c, v * n)  # c1, (v, P)
            Y = Y - cd2 * torch.matmul(a, U.reshape(k, v * n, v)).transpose(1, 2)
    return Y.reshape(k, v * c)


def _dense(M, e, w, v, cx, cd, cd2=0.0, cqp=1.0):
    """The operator as a (v c) x (v c) matrix, rows (v1, c1), columns (v, c)."""
    c = e.numel() - v
    vc = M[:v, :, v:].permute(0, 2, 1).reshape(v * c, -1)  # (vc, P)
    H = torch.zeros((v * c, v * c), dtype=torch.float64, device=M.device)
    if cx:
        H = H + cx * (vc @ vc.T)
    if cd:
        vv = (M[:v, :, :v] * w[None, :, None]).permute(0, 2, 1).reshape(v * v, -1)  # (v1, v), P
        cc = M[v:, :, v:].permute(0, 2, 1).reshape(c * c, -1)  # (c1, c), P
        H = H - cd * (vv @ cc.T).reshape(v, v, c, c).permute(0, 2, 1, 3).reshape(v * c, v * c)
    if cd2:
        cv = (M[v:, :, :v] * w[None, :, None]).permute(0, 2, 1).reshape(c * v, -1)  # (c1, v), P
        H = H - cd2 * (vc @ cv.T).reshape(v, c, c, v).permute(0, 2, 3, 1).reshape(v * c, v * c)
    if cqp:
        H = H + cqp * torch.diag((e[v:][None, :] - e[:v][:, None]).reshape(-1))
    return H


def _roots(H, n):
    return torch.linalg.eigvalsh(0.5 * (H + H.T))[:n].cpu().numpy()


def exact(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind in ("product", "ham"):
        M, e, w = _blocks(seed, case)
        v, dim = case["v"], case["v"] * case["c"]
        if kind == "product":
            cqp, cx, cd = COEF[case["spin"]]
            Y = _apply_exact(M, e, w, v, _vectors(seed, dim, case["k"]), cqp, cx, cd)
            return np.ascontiguousarray(Y.cpu().numpy().T) if case["host"] else Y
        X = _vectors(seed, 2 * dim, case["k"])
        t, b = X[:, :dim], X[:, dim:]
        A = [_apply_exact(M, e, w, v, x, 1.0, 2.0, 1.0) for x in (t, b)]
        B = [_apply_exact(M, e, w, v, x, 0.0, 2.0, 0.0, 1.0) for x in (t, b)]
        return torch.cat([A[0] + B[1], -A[1] - B[0]], dim=1).T.contiguous().cpu().numpy()
    if kind == "solve":
        M, e, w = _blocks(seed, case)
        _, cx, cd = COEF[case["spin"]]
        return dict(evals=_roots(_dense(M, e, w, case["v"], cx, cd), case["roots"]), evecs=None, success=None)
    if kind == "full_solve":
        M, e, w = _blocks(seed, case)
        A = _dense(M, e, w, case["v"], 2.0, 1.0)
        B = _dense(M, e, w, case["v"], 2.0, 0.0, 1.0, cqp=0.0)
        L = torch.linalg.cholesky(A - B)
        return dict(evals=np.sqrt(_roots(L.T @ (A + B) @ L, case["roots"])), X=None, Y=None, success=None)
    if kind == "batch":
        _, cx, cd = COEF[case["spin"]]
        evals, cost = [], 0.0
        for v, c, naux, sd in _batch_shapes(case, seed):
            cost += (v * c) ** 3
        if cost > 4e12:
            return None
        for v, c, naux, sd in _batch_shapes(case, seed):
            M, e, w = _blocks(sd, dict(v=v, c=c, naux=naux))
            evals.append(_roots(_dense(M, e, w, v, cx, cd), case["roots"]))
        return dict(evals=np.stack(evals), success=None)
    if kind == "gradient":
        v, c, r = case["v"], case["c"], case["roots"]
        M, e, w = _blocks(seed, case)
        H = _dense(M, e, w, v, 2.0, 1.0)
        lam, U = torch.linalg.eigh(0.5 * (H + H.T))
        x = U[:, :r].T.reshape(r, v, c)
        M, w = M.requires_grad_(True), w.requires_grad_(True)
        h = torch.diag(e).requires_grad_(True)
        g = torch.linspace(1.0, 2.0, r, dtype=torch.float64, device="cuda")
        # sum_k g_k x_k^T H x_k with the eigenvectors fixed (Hellmann-Feynman)
        z = torch.einsum("kvc,vpc->kp", x, M[:v, :, v:])
        S = torch.einsum("kvc,dpc->kvpd", x, M[v:, :, v:])
        f = (g[:, None] * 2.0 * z * z).sum()
        f = f - torch.einsum("k,kud,upv,p,kvpd->", g, x, M[:v, :, :v], w, S)
        f = f + torch.einsum("k,kvc,cd,kvd->", g, x, h[v:, v:], x) - torch.einsum("k,kvc,uv,kuc->", g, x, h[:v, :v], x)
        f.backward()
        return dict(evals=lam[:r].detach(), mmn=M.grad, hqp=h.grad, w=w.grad)
    if kind == "screening":
        v = case["v"]
        M, e, _ = _blocks(seed, case)
        dE = (e[v:][None, :] - e[:v][:, None]).reshape(-1)
        B = M[:v, :, v:].permute(0, 2, 1).reshape(dE.numel(), -1)
        chi = -2.0 * dE / (dE * dE + 1e-8)  # at zero frequency, with the small broadening of the RPA
        eps = torch.eye(case["naux"], dtype=torch.float64, device="cuda") - 2.0 * (B.T @ (chi[:, None] * B))
        return dict(eps=eps.cpu().numpy(), W=torch.linalg.inv(eps).cpu().numpy())
    ao, C, U = _ao_inputs(seed, case["nbf"], case["nmo"], case["naux"])
    M = torch.matmul(torch.matmul(C.T, ao), C)  # (P, m, n)
    return torch.einsum("pmn,pq->mqn", M, U).contiguous().cpu().numpy()
