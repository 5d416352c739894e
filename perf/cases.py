"""The work that users of this framework have it do, as timed cases through its public API.

Every case is a dict of plain values with a `kind`:

  mult       C = beta*C + alpha*op(A)*op(B)                        (Mult)
  chol       factor an SPD matrix and solve with it, FP64          (DecomposeCHOL, SolveCHOL)
  lu         factor a general matrix with pivoting and solve       (DecomposeLU, SolveLU)
  mixed      SPD solve, split-product factor + FP64 refinement     (SolveCHOLMixed)
  batch      factor + solve many small systems of uneven order     (BatchPlan.run)
  chol_grad  Cholesky of many equal matrices, forward and reverse  (BatchPlan.run,
             DecomposeCHOLAdjointBatched)
  lstsq      least squares by QR in the compact WY form            (DecomposeQRT, SolveQRT)

The factorizations work in place, so a pass starts by copying the caller's matrix into the
work matrix, as a program that needs its matrix again does.
"""
import math

import numpy as np
import torch

import matops_b200 as mo

F64 = torch.float64


def listed():
    return [
        # one small product inside a host loop: launch and call latency
        {"name": "mult_64", "kind": "mult", "m": 64, "n": 64, "k": 64, "pad": 0, "flags": 0,
         "alpha": 1.0, "beta": 0.0},
        # the plain DGEMM of the benchmark
        {"name": "mult_2048", "kind": "mult", "m": 2048, "n": 2048, "k": 2048, "pad": 0,
         "flags": 0, "alpha": 1.5, "beta": -0.5},
        # a product of odd sizes with a transposed operand and odd leading dimensions
        {"name": "mult_ragged_t", "kind": "mult", "m": 3001, "n": 1777, "k": 2503, "pad": 0,
         "flags": mo.TRANSA, "alpha": 1.0, "beta": 1.0},
        # one SPD system of a few hundred unknowns (a Gaussian-process fit, a Kalman update)
        {"name": "chol_500", "kind": "chol", "n": 500, "nrhs": 1, "flags": mo.LOWER},
        # the benchmark's FP64 Cholesky solve
        {"name": "chol_16384", "kind": "chol", "n": 16384, "nrhs": 64, "flags": mo.LOWER},
        # a general system of about a thousand unknowns, odd order
        {"name": "lu_1001", "kind": "lu", "n": 1001, "nrhs": 3},
        # the benchmark's LU solve
        {"name": "lu_16384", "kind": "lu", "n": 16384, "nrhs": 64},
        # the benchmark's headline: mixed-precision Cholesky solve refined to 1e-14
        {"name": "mixed_16384", "kind": "mixed", "n": 16384, "nrhs": 64, "flags": mo.LOWER,
         "prec": mo.PREC_BF16X3},
        # the benchmark's batches of small systems
        {"name": "batch_chol_4096", "kind": "batch", "method": "chol", "count": 4096,
         "nmin": 16, "nmax": 512, "nrhs": 1},
        {"name": "batch_lu_4096", "kind": "batch", "method": "lu", "count": 4096, "nmin": 16,
         "nmax": 512, "nrhs": 1},
        # the benchmark's differentiated batch: forward and reverse sweep
        {"name": "chol_grad_512x256", "kind": "chol_grad", "count": 512, "n": 256},
        # a tall regression with a few targets
        {"name": "lstsq_8000x2000", "kind": "lstsq", "m": 8000, "n": 2000, "nrhs": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mult", "chol", "lu", "mixed", "batch", "batch", "chol_grad", "lstsq"])
    nrhs = rng.choice([1, 2, 3, 8, 16, 31, 64])
    if kind == "mult":
        return {"kind": kind, "m": _log(rng, 16, 4096), "n": _log(rng, 16, 4096),
                "k": _log(rng, 16, 4096), "pad": rng.choice([0, 0, 1, 2, 7]),
                "flags": rng.choice([0, mo.TRANSA, mo.TRANSB, mo.TRANSA | mo.TRANSB]),
                "alpha": rng.choice([1.0, -1.0, 1.5]), "beta": rng.choice([0.0, 1.0, -0.5])}
    if kind == "chol":
        return {"kind": kind, "n": _log(rng, 64, 16384), "nrhs": nrhs,
                "flags": rng.choice([mo.LOWER, mo.LOWER, mo.UPPER])}
    if kind == "lu":
        return {"kind": kind, "n": _log(rng, 64, 12000), "nrhs": nrhs}
    if kind == "mixed":
        return {"kind": kind, "n": _log(rng, 512, 16384), "nrhs": nrhs,
                "flags": rng.choice([mo.LOWER, mo.LOWER, mo.UPPER]),
                "prec": rng.choice([mo.PREC_BF16X3, mo.PREC_TF32X3])}
    if kind == "batch":
        nmin = _log(rng, 8, 200)
        return {"kind": kind, "method": rng.choice(["chol", "lu"]),
                "count": _log(rng, 128, 4096), "nmin": nmin,
                "nmax": rng.randint(nmin, 512), "nrhs": rng.choice([1, 1, 2, 5])}
    if kind == "chol_grad":
        n = _log(rng, 24, 512)
        return {"kind": kind, "count": rng.randint(32, 512), "n": n}
    m = _log(rng, 128, 8192)
    return {"kind": kind, "m": m, "n": max(1, int(m * rng.uniform(0.05, 0.6))), "nrhs": nrhs}


# ---- inputs ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 + int(seed))


def _mat(r, c, pad=0):
    """an uninitialized column-major r x c matrix with leading dimension r + pad"""
    return mo.matrix(r + pad, c)[:r]


def _normal(r, c, g, pad=0):
    t = mo.matrix(r + pad, c)
    t.normal_(generator=g)
    return t[:r]


def _uniform(r, c, g, pad=0):
    t = mo.matrix(r + pad, c)
    t.uniform_(-1.0, 1.0, generator=g)
    return t[:r]


def _spd(n, g, shift):
    """G G^T / n + shift*I, symmetric to the bit, column-major"""
    G = torch.randn(n, n, dtype=F64, device="cuda", generator=g)
    A = torch.mm(G, G.t()).div_(n)
    del G
    A = torch.tril(A) + torch.tril(A, -1).t()
    A.diagonal().add_(shift)
    return A.t()


def _batch_orders(case):
    """the plan's orders belong to the case, like the shape of a single matrix"""
    rng = np.random.default_rng([case["count"], case["nmin"], case["nmax"]])
    return rng.integers(case["nmin"], case["nmax"] + 1, case["count"]).astype(np.int32)


def _offsets(sizes, unit):
    """start of each piece of sizes[i] elements, every one on a multiple of `unit`"""
    padded = -(-sizes.astype(np.int64) // unit) * unit
    return np.concatenate([[0], np.cumsum(padded)])


def _batch_inputs(case, seed):
    """orders, and the flat buffers of matrices and right-hand sides with their offsets"""
    n = _batch_orders(case)
    g = _gen(seed)
    ao = _offsets(n.astype(np.int64) ** 2, 32)
    bo = _offsets(n.astype(np.int64) * case["nrhs"], 32)
    A = torch.zeros(int(ao[-1]), dtype=F64, device="cuda")
    B = torch.randn(int(bo[-1]), dtype=F64, device="cuda", generator=g)
    A.normal_(generator=g)
    if case["method"] == "chol":
        for a in _pieces(A, ao, n):
            s = torch.mm(a, a.t()).div_(a.shape[0])
            s.diagonal().add_(1.0)
            a.copy_(s)
    return n, ao, bo, A, B


def _pieces(flat, offs, n, cols=None):
    """the column-major matrices of a flat buffer: n[i] x n[i], or n[i] x cols"""
    out = []
    for i, k in enumerate(n.tolist()):
        c = k if cols is None else cols
        out.append(torch.as_strided(flat, (k, c), (1, k), int(offs[i])))
    return out


def _grad_inputs(case, seed):
    g = _gen(seed)
    n, count = case["n"], case["count"]
    G = torch.randn(count, n, n, dtype=F64, device="cuda", generator=g)
    A = torch.bmm(G, G.transpose(1, 2)).div_(n)
    A = torch.tril(A) + torch.tril(A, -1).transpose(1, 2)
    A.diagonal(dim1=1, dim2=2).add_(1.0)
    W = torch.tril(torch.randn(count, n, n, dtype=F64, device="cuda", generator=g))
    return A, W


def _inputs(case, seed):
    """the plain inputs of the single-matrix kinds"""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "mult":
        m, n, k, f, pad = case["m"], case["n"], case["k"], case["flags"], case["pad"]
        A = _uniform(*((k, m) if f & mo.TRANSA else (m, k)), g, pad)
        B = _uniform(*((n, k) if f & mo.TRANSB else (k, n)), g, pad)
        return A, B, _uniform(m, n, g, pad)
    if kind in ("chol", "mixed"):
        return _spd(case["n"], g, 0.5), _uniform(case["n"], case["nrhs"], g)
    if kind == "lu":
        return _normal(case["n"], case["n"], g), _uniform(case["n"], case["nrhs"], g)
    return _normal(case["m"], case["n"], g), _uniform(case["m"], case["nrhs"], g)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        n, ao, bo, A0, B0 = _batch_inputs(case, seed)
        A, B = torch.empty_like(A0), torch.empty_like(B0)
        s.update(A0=A0, B0=B0, A=A, B=B, As=_pieces(A, ao, n),
                 Bs=_pieces(B, bo, n, case["nrhs"]), piv=None, pivs=None)
        chol = case["method"] == "chol"
        if not chol:
            po = np.concatenate([[0], np.cumsum(n.astype(np.int64))])
            s["piv"] = torch.zeros(int(po[-1]), dtype=torch.int64, device="cuda")
            s["pivs"] = [s["piv"][int(po[i]):int(po[i + 1])] for i in range(len(n))]
        s["plan"] = mo.BatchPlan(mo.BATCH_CHOL if chol else mo.BATCH_LU, n, case["nrhs"])
    elif kind == "chol_grad":
        A0, W = _grad_inputs(case, seed)
        L, Lb = torch.empty_like(A0), torch.empty_like(W)
        # W as column-major matrices: element (i, r, c) at [i, c, r] of the buffer
        s.update(A0=A0, W=W.transpose(1, 2).contiguous(), L=L, Lb=Lb,
                 Ls=[t.t() for t in L], Lbs=[t.t() for t in Lb],
                 plan=mo.BatchPlan(mo.BATCH_CHOL, [case["n"]] * case["count"], 0))
    elif kind == "mult":
        A, B, C0 = _inputs(case, seed)
        s.update(A=A, B=B, C0=C0, C=_mat(case["m"], case["n"], case["pad"]))
        s["C"].copy_(C0)
    else:
        A0, B0 = _inputs(case, seed)
        s.update(A0=A0, B0=B0, B=torch.empty_like(B0))
        if kind == "mixed":
            s["X"] = s["B"]
        else:
            s["A"] = torch.empty_like(A0)
        if kind == "lu":
            s["piv"] = torch.zeros(case["n"], dtype=torch.int64, device="cuda")
        if kind == "lstsq":
            s["T"] = mo.matrix(case["n"], case["n"], fill=0.0)
            s["W"] = mo.matrix(case["nrhs"], case["n"])
    return s


# ---- one pass -------------------------------------------------------------------------

def _ok(err):
    if err is not None:
        raise err


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mult":
        if case["beta"] != 0.0:
            s["C"].copy_(s["C0"])
        _ok(mo.Mult(s["C"], s["A"], s["B"], case["alpha"], case["beta"], case["flags"]))
        return s["C"]
    if kind == "chol":
        s["A"].copy_(s["A0"])
        s["B"].copy_(s["B0"])
        _ok(mo.DecomposeCHOL(s["A"], case["flags"], 0)[1])
        mo.SolveCHOL(s["B"], s["A"], case["flags"])
        return s["A"], s["B"]
    if kind == "lu":
        s["A"].copy_(s["A0"])
        s["B"].copy_(s["B0"])
        _ok(mo.DecomposeLU(s["A"], s["piv"], 0)[1])
        _ok(mo.SolveLU(s["B"], s["A"], s["piv"], mo.NONE))
        return s["A"], s["B"], s["piv"]
    if kind == "mixed":
        info, err = mo.SolveCHOLMixed(s["X"], s["A0"], s["B0"], case["flags"], case["prec"])
        _ok(err)
        return s["X"]
    if kind == "batch":
        s["A"].copy_(s["A0"])
        s["B"].copy_(s["B0"])
        info = s["plan"].run(s["As"], s["Bs"], s["pivs"])
        if s["piv"] is None:
            return s["A"], s["B"], info
        return s["A"], s["B"], info, s["piv"]
    if kind == "chol_grad":
        s["L"].copy_(s["A0"])
        s["Lb"].copy_(s["W"])
        info = s["plan"].run(s["Ls"])
        _ok(mo.DecomposeCHOLAdjointBatched(s["Ls"], s["Lbs"], mo.LOWER))
        return s["L"], s["Lb"], info
    s["A"].copy_(s["A0"])
    s["B"].copy_(s["B0"])
    _ok(mo.DecomposeQRT(s["A"], s["T"], None, 0)[1])
    _ok(mo.SolveQRT(s["B"], s["A"], s["T"], s["W"], mo.NONE, 0))
    return s["A"], s["T"], s["B"]


# ---- what a pass cannot do without ------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "mult":
        m, n, k = case["m"], case["n"], case["k"]
        c = 2 if case["beta"] != 0.0 else 1
        return {"bytes": 8.0 * (m * k + k * n + c * m * n), "flops": 2.0 * m * n * k}
    if kind in ("chol", "lu", "mixed"):
        n, r = float(case["n"]), case["nrhs"]
        # a triangle in (and its factor out) for SPD; the whole matrix in and out for LU
        elems = {"chol": n * n, "lu": 2.0 * n * n, "mixed": n * n / 2}[kind]
        fact = 2.0 * n ** 3 / 3.0 if kind == "lu" else n ** 3 / 3.0
        return {"bytes": 8.0 * (elems + 2.0 * n * r), "flops": fact + 2.0 * n * n * r}
    if kind == "batch":
        n = _batch_orders(case).astype(np.float64)
        lu = case["method"] == "lu"
        fl = ((2.0 if lu else 1.0) * n ** 3 / 3.0 + 2.0 * n * n * case["nrhs"]).sum()
        by = 8.0 * ((2.0 if lu else 1.0) * n * n + 2.0 * n * case["nrhs"]).sum()
        return {"bytes": float(by), "flops": float(fl)}
    if kind == "chol_grad":
        n, c = float(case["n"]), case["count"]
        # A's triangle in, L out, Lbar's triangle in, the symmetric gradient out
        return {"bytes": 8.0 * c * 2.5 * n * n, "flops": c * n ** 3}
    m, n, r = float(case["m"]), float(case["n"]), case["nrhs"]
    return {"bytes": 8.0 * (2.0 * m * n + n * n / 2 + 2.0 * m * r),
            "flops": 2.0 * m * n * n - 2.0 * n ** 3 / 3.0      # R and the reflectors
            + m * n * n - n ** 3 / 3.0                         # T
            + 4.0 * m * n * r + n * n * r}                     # Q^T B and the R solve


# ---- the same in plain torch, 64 bits ---------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        n, ao, bo, A, B = _batch_inputs(case, seed)
        pivs = []
        for a, b in zip(_pieces(A, ao, n), _pieces(B, bo, n, case["nrhs"])):
            if case["method"] == "chol":
                L = torch.linalg.cholesky_ex(a)[0]
                b.copy_(torch.cholesky_solve(b, L))
                a.copy_(torch.tril(L) + torch.triu(a, 1))
            else:
                LU, p = torch.linalg.lu_factor(a)
                b.copy_(torch.linalg.lu_solve(LU, p, b))
                a.copy_(LU)
                pivs.append(p.to(torch.int64) - 1)
        info = None
        return (A, B, info) if case["method"] == "chol" else (A, B, info, torch.cat(pivs))
    if kind == "chol_grad":
        A, W = _grad_inputs(case, seed)
        A.requires_grad_(True)
        L = torch.linalg.cholesky(A)
        L.backward(W)
        full = torch.tril(L.detach()) + torch.triu(A.detach(), 1)
        return full.transpose(1, 2), A.grad.transpose(1, 2), None
    if kind == "mult":
        A, B, C = _inputs(case, seed)
        f = case["flags"]
        P = torch.mm(A.t() if f & mo.TRANSA else A, B.t() if f & mo.TRANSB else B)
        return case["alpha"] * P + case["beta"] * C
    A, B = _inputs(case, seed)
    if kind == "chol":
        L = torch.linalg.cholesky(A)
        X = torch.cholesky_solve(B, L)
        if case["flags"] & mo.UPPER:
            return torch.triu(L.t()) + torch.tril(A, -1), X
        return torch.tril(L) + torch.triu(A, 1), X
    if kind == "mixed":
        return torch.cholesky_solve(B, torch.linalg.cholesky(A))
    if kind == "lu":
        LU, p = torch.linalg.lu_factor(A)
        return LU, torch.linalg.lu_solve(LU, p, B), p.to(torch.int64) - 1
    n = case["n"]
    QR, tau = torch.geqrf(A)
    V = torch.tril(QR, -1)
    V.diagonal().fill_(1.0)
    # the block reflector T of Q = I - V T V^T: T^-1 = triu(V^T V, 1) + diag(1 / tau)
    Ti = torch.triu(torch.mm(V.t(), V), 1)
    Ti.diagonal().copy_(1.0 / tau)
    T = torch.linalg.solve_triangular(Ti, torch.eye(n, dtype=F64, device=A.device), upper=True)
    C = B - torch.mm(V, torch.mm(T.t(), torch.mm(V.t(), B)))
    X = torch.linalg.solve_triangular(QR[:n], C[:n], upper=True)
    return QR, T, torch.cat([X, C[n:]])
