"""Performance cases of the QR path: what its users run, through the public entry points.

A case is a dict of plain values; its "kind" names the entry points:

  panel    hh_recon_qr: TSQR and Householder reconstruction of one tall-skinny panel
  tsqr     bitree_tsqr, then construct_Q1: R and an explicit orthonormal basis
  update   upd_A: the compact-WY trailing update A <- (I - Y T Y^T)^T A
  caqr     QR_2D / QR_2D_pipe: blocked factorization of a matrix
  ls       ls_solve: least squares with FP64 refinement
  batch    batched_ls / batched_ls_f32: many independent tall-skinny problems
  serve    LSServer: a burst of least-squares requests held in host memory

Entries are iid N(0, 1), the distribution of the benchmark's panels, batches and
requests; the columns of the "caqr" matrices are graded over three decades.
"""
import math

import numpy as np
import torch

import candmc_gb300 as cm
from candmc_gb300.serve import LSServer

WIDTHS_BATCH = (8, 16, 32, 64, 128)
WIDTHS_SERVE = (16, 32, 64, 128, 256)
SERVE_WORKERS = 8
SERVE_POOL = 18_000_000   # doubles of host memory that the requests' matrices are slices of


def listed():
    return [
        # one small panel: the latency of a single call
        {"name": "panel 512x32", "kind": "panel", "m": 512, "b": 32},
        # the panel of the benchmark's TSQR-HR configuration
        {"name": "panel 8192x64", "kind": "panel", "m": 8192, "b": 64},
        # a tall panel with ragged row blocks and an odd width
        {"name": "panel 100003x99", "kind": "panel", "m": 100003, "b": 99},
        # an orthonormal basis of a tall block of vectors, as block Krylov methods need it
        {"name": "tsqr 65537x48", "kind": "tsqr", "m": 65537, "b": 48},
        # one trailing update of a blocked factorization that drives its own panels
        {"name": "update 8192x4096x128 ozaki", "kind": "update", "m": 8192, "n": 4096, "b": 128,
         "precision": "ozaki", "w": "none"},
        # a small dense factorization in plain FP64
        {"name": "caqr 1500x1000 fp64", "kind": "caqr", "entry": "QR_2D", "m": 1500, "n": 1000, "b": 64,
         "precision": "fp64"},
        # a mid-sized factorization of odd sizes in the tensor-core form
        {"name": "caqr 4097x4001 ozaki", "kind": "caqr", "entry": "QR_2D_pipe", "m": 4097, "n": 4001, "b": 128,
         "precision": "ozaki"},
        # the benchmark's square factorization
        {"name": "caqr 16384x16384 ozaki", "kind": "caqr", "entry": "QR_2D_pipe", "m": 16384, "n": 16384,
         "b": 128, "precision": "ozaki"},
        # one tall regression, factored in the FP32 form and refined to FP64
        {"name": "ls 262144x128 fp32", "kind": "ls", "m": 262144, "n": 128, "nrhs": 1, "precision": "fp32"},
        # a larger system with several right-hand sides
        {"name": "ls 16384x4096x16 ozaki", "kind": "ls", "m": 16384, "n": 4096, "nrhs": 16, "precision": "ozaki"},
        # a batch of uneven problems under a captured schedule
        {"name": "batch 128 f64", "kind": "batch", "count": 128, "m_lo": 256, "m_hi": 65536, "sizes": 3,
         "dtype": "f64", "graph": True},
        # requests that arrive together at the server
        {"name": "serve 24", "kind": "serve", "count": 24, "m_lo": 512, "m_hi": 65536, "sizes": 4,
         "precision": "fp32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["panel", "panel", "tsqr", "update", "caqr", "caqr", "ls", "ls", "batch", "serve"])
    if kind in ("panel", "tsqr"):
        b = _log(rng, 8, 128)
        return {"kind": kind, "m": max(b, _log(rng, 256, 262144)), "b": b}
    if kind == "update":
        b = rng.choice([32, 64, 128, rng.randint(17, 127)])
        return {"kind": kind, "m": max(b, _log(rng, 512, 16384)), "n": _log(rng, 64, 8192), "b": b,
                "precision": rng.choice(["ozaki", "fp64"]), "w": rng.choice(["none", "T"])}
    if kind == "caqr":
        p = rng.choice(["ozaki", "ozaki", "fp64"])
        n = _log(rng, 128, 6000 if p == "ozaki" else 2500)
        return {"kind": kind, "entry": rng.choice(["QR_2D", "QR_2D_pipe"]), "m": int(n * math.exp(rng.uniform(0.0, 1.2))),
                "n": n, "b": rng.choice([32, 64, 128]), "precision": p}
    if kind == "ls":
        n = _log(rng, 16, 512)
        return {"kind": kind, "m": max(2 * n, _log(rng, 512, 2 ** 27 // n if n > 128 else 2 ** 20)), "n": n,
                "nrhs": rng.choice([1, 1, 16, rng.randint(2, 15)]), "precision": rng.choice(["fp32", "ozaki", "fp64"])}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 8, 128), "m_lo": 256, "m_hi": _log(rng, 2048, 65536),
                "sizes": rng.randint(5, 10 ** 6), "dtype": rng.choice(["f64", "f32"]), "graph": rng.random() < 0.5}
    return {"kind": kind, "count": rng.randint(6, 24), "m_lo": 512, "m_hi": _log(rng, 4096, 65536),
            "sizes": rng.randint(5, 10 ** 6), "precision": rng.choice(["fp32", "fp64"])}


def _sizes(case, widths):
    """The uneven (m, n) of a batch or a burst: m log-uniform, n uniform over the widths."""
    rng = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["count"]):
        m = int(round(math.exp(rng.uniform(math.log(case["m_lo"]), math.log(case["m_hi"])))))
        n = int(rng.choice(widths))
        out.append((max(m, 2 * n), n))
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(m, n, g, dtype=torch.float64):
    """Column-major m x n with iid N(0, 1) entries."""
    return torch.randn(n, m, dtype=dtype, device="cuda", generator=g).t()


def _matrix(case, seed):
    if case["kind"] == "caqr":
        A = _normal(case["m"], case["n"], _gen(seed))
        A *= torch.logspace(0, -3, case["n"], dtype=torch.float64, device="cuda")
        return A
    return _normal(case["m"], case["b"], _gen(seed))


def _update_inputs(case, seed):
    g = _gen(seed)
    m, b = case["m"], case["b"]
    # reflectors of a random panel: unit lower trapezoidal, tails of norm about one
    Y = _normal(m, b, g) / math.sqrt(m)
    top = torch.tril(Y[:b], -1) + torch.eye(b, dtype=torch.float64, device="cuda")
    Y[:b] = top
    return Y, _normal(m, case["n"], g)


def _invT(Y):
    """T^-T of the compact-WY form: the lower part of Y^T Y with its diagonal halved."""
    G = Y.t() @ Y
    return torch.tril(G, -1) + torch.diag(G.diagonal() / 2)


def _batch_layout(sizes):
    """Offsets of every A_i and b_i in two flat buffers, 32 elements aligned."""
    offa, offb, ta, tb = [], [], 0, 0
    for m, n in sizes:
        offa.append(ta)
        offb.append(tb)
        ta += -(-m * n // 32) * 32
        tb += -(-m // 32) * 32
    return offa, offb, ta, tb


def _batch_views(sizes, offa, offb, fa, fb):
    As = [fa[o:o + m * n].view(n, m).t() for (m, n), o in zip(sizes, offa)]
    Bs = [fb[o:o + m].view(1, m).t() for (m, n), o in zip(sizes, offb)]
    return As, Bs


def _batch_inputs(case, seed):
    sizes = _sizes(case, WIDTHS_BATCH)
    offa, offb, ta, tb = _batch_layout(sizes)
    g = _gen(seed)
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    return sizes, offa, offb, torch.randn(ta, dtype=dt, device="cuda", generator=g), \
        torch.randn(tb, dtype=dt, device="cuda", generator=g)


def _serve_inputs(case, seed):
    """Host matrices as slices of one pool, (A_i, b_i) of every request."""
    pool = np.random.default_rng(seed).standard_normal(SERVE_POOL)
    out, at = [], 0
    for i, (m, n) in enumerate(_sizes(case, WIDTHS_SERVE)):
        at = (at + 7919 * (i + 1)) % (SERVE_POOL - m * (n + 1))
        out.append((pool[at:at + m * n].reshape(n, m).T, pool[at + m * n:at + m * n + m]))
    return out


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("panel", "tsqr", "caqr"):
        st["A0"] = _matrix(case, seed)
        st["A"] = torch.empty_like(st["A0"])
    elif kind == "update":
        st["Y"], st["A0"] = _update_inputs(case, seed)
        st["A"] = torch.empty_like(st["A0"])
        st["W"] = cm.colmajor(_invT(st["Y"])) if case["w"] == "T" else None
    elif kind == "ls":
        g = _gen(seed)
        st["A"] = _normal(case["m"], case["n"], g)
        st["B"] = _normal(case["m"], case["nrhs"], g)
    elif kind == "batch":
        sizes, offa, offb, st["fa0"], st["fb0"] = _batch_inputs(case, seed)
        st["fa"], st["fb"] = torch.empty_like(st["fa0"]), torch.empty_like(st["fb0"])
        st["As"], st["Bs"] = _batch_views(sizes, offa, offb, st["fa"], st["fb"])
    else:
        st["requests"] = _serve_inputs(case, seed)
        st["server"] = LSServer(workers=SERVE_WORKERS, precision=case["precision"])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "panel":
        # the caller keeps its matrix: the factorization works on a copy
        st["A"].copy_(st["A0"])
        W, T = cm.hh_recon_qr(st["A"])
        return {"YR": st["A"], "W": W, "T": T}
    if kind == "tsqr":
        st["A"].copy_(st["A0"])
        R, tau = cm.bitree_tsqr(st["A"])
        return {"YR": st["A"], "R": R, "tau": tau, "Q1": cm.construct_Q1(st["A"], tau)}
    if kind == "update":
        st["A"].copy_(st["A0"])
        cm.upd_A(st["Y"], st["A"], W=st["W"], W_is_T=st["W"] is not None, precision=case["precision"])
        return {"A": st["A"]}
    if kind == "caqr":
        st["A"].copy_(st["A0"])
        getattr(cm, case["entry"])(st["A"], case["b"], precision=case["precision"])
        return {"YR": st["A"]}
    if kind == "ls":
        X, _ = cm.ls_solve(st["A"], st["B"], precision=case["precision"])
        return {"X": X}
    if kind == "batch":
        st["fa"].copy_(st["fa0"])
        st["fb"].copy_(st["fb0"])
        solve = cm.batched_ls if case["dtype"] == "f64" else cm.batched_ls_f32
        solve(st["As"], st["Bs"], use_graph=case["graph"])
        # f64: Y\R of every problem too; f32 leaves the matrices as they were
        return {"B": st["fb"], "A": st["fa"]}
    srv = st["server"]
    tickets = [srv.submit(A, b) for A, b in st["requests"]]
    return {"x": np.concatenate([srv.result(t)[0] for t in tickets])}


def _qr_flops(m, n):
    return 2.0 * n * n * (m - n / 3.0)


def work(case):
    kind = case["kind"]
    if kind == "panel":
        m, b = case["m"], case["b"]
        return {"bytes": 16.0 * m * b, "flops": _qr_flops(m, b) + 1.0 * m * b * b}
    if kind == "tsqr":
        m, b = case["m"], case["b"]
        return {"bytes": 24.0 * m * b, "flops": 2 * _qr_flops(m, b)}
    if kind == "update":
        m, n, b = case["m"], case["n"], case["b"]
        return {"bytes": 8.0 * (m * b + 2 * m * n), "flops": 4.0 * m * n * b}
    if kind == "caqr":
        return {"bytes": 16.0 * case["m"] * case["n"], "flops": _qr_flops(case["m"], case["n"])}
    if kind == "ls":
        m, n, r = case["m"], case["n"], case["nrhs"]
        return {"bytes": 8.0 * (m * n + m * r + n * r), "flops": _qr_flops(m, n) + 4.0 * m * n * r}
    if kind == "batch":
        sizes, w = _sizes(case, WIDTHS_BATCH), (16.0 if case["dtype"] == "f64" else 4.0)
    else:
        sizes, w = _sizes(case, WIDTHS_SERVE), 8.0
    return {"bytes": sum(w * m * n + 8.0 * (m + n) for m, n in sizes),
            "flops": sum(_qr_flops(m, n) + 4.0 * m * n for m, n in sizes)}


def _house(A):
    """(Y\\R, tau) of LAPACK's Householder QR.  The last reflector of a square
    matrix has an empty tail: here it is a sign flip (tau = 2), there the identity."""
    a, tau = torch.geqrf(A)
    if A.shape[0] == A.shape[1]:
        a[-1, -1] = -a[-1, -1]
        tau[-1] = 2.0
    return a, tau


def _unit_lower(a):
    m, n = a.shape
    return torch.tril(a, -1) + torch.eye(m, n, dtype=a.dtype, device=a.device)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("panel", "tsqr", "caqr"):
        A = _matrix(case, seed)
        if kind == "caqr":
            return {"YR": _house(A)[0]}
        a, tau = _house(A)
        b = case["b"]
        Y = _unit_lower(a)
        if kind == "panel":
            T = torch.linalg.inv(_invT(Y)).t()
            return {"YR": a, "W": torch.triu(-T @ Y[:b].t()), "T": torch.triu(T)}
        T = torch.linalg.inv(_invT(Y)).t()
        Q1 = -Y @ (T @ Y[:b].t())
        Q1[:b] += torch.eye(b, dtype=torch.float64, device="cuda")
        return {"YR": a, "R": torch.triu(a[:b]), "tau": tau, "Q1": Q1}
    if kind == "update":
        Y, A = _update_inputs(case, seed)
        return {"A": A - Y @ torch.linalg.solve_triangular(_invT(Y), Y.t() @ A, upper=False)}
    if kind == "ls":
        g = _gen(seed)
        A = _normal(case["m"], case["n"], g)
        return {"X": _solve(A, _normal(case["m"], case["nrhs"], g))}
    if kind == "batch":
        sizes, offa, offb, fa, fb = _batch_inputs(case, seed)
        f64 = case["dtype"] == "f64"
        da, db = fa.double(), fb.double()
        As, Bs = _batch_views(sizes, offa, offb, da, db)
        for A, B in zip(As, Bs):
            n = A.shape[1]
            if f64:
                a, tau = _house(A)
                Y = _unit_lower(a)
                B -= Y @ (torch.linalg.solve_triangular(_invT(Y), Y.t() @ B, upper=False))
                A.copy_(a)
                B[:n] = torch.linalg.solve_triangular(torch.triu(a[:n]), B[:n], upper=True)
            else:
                B[:n] = _solve(A, B)
        return {"B": db if f64 else db.float(), "A": da if f64 else fa}
    xs = []
    for A, b in _serve_inputs(case, seed):
        A = torch.from_numpy(np.ascontiguousarray(A)).cuda()
        xs.append(_solve(A, torch.from_numpy(np.ascontiguousarray(b)).cuda().view(-1, 1))[:, 0])
    return {"x": torch.cat(xs).cpu().numpy()}


def _solve(A, B):
    """min ||A X - B|| from the QR of [A | B], with one correction of its residual."""
    n = A.shape[1]
    a, _ = torch.geqrf(torch.cat([A, B], 1) if A.shape[0] > n + B.shape[1] else A)
    R = torch.triu(a[:n, :n])
    X = torch.zeros(n, B.shape[1], dtype=torch.float64, device=A.device)
    for _ in range(4):
        S = torch.linalg.solve_triangular(R.t(), A.t() @ (B - A @ X), upper=False)
        X = X + torch.linalg.solve_triangular(R, S, upper=True)
    return X
