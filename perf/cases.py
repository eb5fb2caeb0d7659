"""The calls of the tensor-train sweeps that are timed, over the sizes users run.

Every case is one call (or the pair of calls a sweep always makes together)
of the ``ttgpu`` package, on inputs of the values and shapes the sweeps meet:

  apply   LocalOp.apply: the local product y = Phi1 A Phi2 x of a prepared
          local problem, FP64 ("plain") or BF16x3 ("split"); the operator core
          is that of a spin chain (n = 2, rank 5) or of a Laplacian with a
          potential on a grid (n = 16..64, rank 3)
  phi     phi_left and phi_right: the interface updates after a core moved
  zapply  zbfun3 and its adjoint: the products of the complex time stepper
  qr      dqr of a core unfolded to (r n) x r
  svd     dgesvd of a local block with the graded spectrum of a sweep
  eigb    tt_eigb, the block eigensolver, on an XXZ chain
  ksl     ztt_ksl, steps of the complex time stepper
  amen    dtt_amen_solve, the linear solver, on the grid operator

All arrays are flat and column-major.  Random numbers come from the case's
seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "tt-fort_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "tt-fort_gb300"))

import ttgpu  # noqa: E402
from ttgpu import operators  # noqa: E402

DEV = "cuda"
_ctx = None


def _driver_ctx():
    """One library context for the driver calls, kept as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = ttgpu.Context(0)
    return _ctx


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest local products: cores near a chain's ends, or early
        # sweeps of a low rank; a few vectors of a Davidson block
        {"name": "apply_chain_r16", "kind": "apply", "op": "chain", "method": "plain",
         "r1": 16, "n": 2, "r2": 16, "nvec": 4},
        # the middle bonds of the d = 20 Heisenberg chain, block of 5
        {"name": "apply_chain_r64", "kind": "apply", "op": "chain", "method": "plain",
         "r1": 64, "n": 2, "r2": 64, "nvec": 5},
        # the middle bonds of the d = 100 XXZ chain, block of 8
        {"name": "apply_chain_r256", "kind": "apply", "op": "chain", "method": "plain",
         "r1": 256, "n": 2, "r2": 256, "nvec": 8},
        # the tensor-core product of the chosen eigensolver, d = 20 chain
        {"name": "split_chain_r64", "kind": "apply", "op": "chain", "method": "split",
         "r1": 64, "n": 2, "r2": 64, "nvec": 5},
        # interface updates of the d = 10, n = 64 grid solve at the ranks it
        # reaches (82 and, after a truncation, an odd one)
        {"name": "phi_grid_r82", "kind": "phi", "op": "grid", "r1": 82, "n": 64, "r2": 77},
        # operator and adjoint of the time stepper at a rank that grew, with
        # the block of four of its norm estimate
        {"name": "zapply_r48", "kind": "zapply", "r1": 48, "n": 32, "r2": 48, "nvec": 4},
        # orthogonalisation of a grid core with its enrichment columns
        {"name": "qr_grid_5248x86", "kind": "qr", "rows": 5248, "cols": 86},
        # truncation of a local block of the d = 20 chain: (B r) x (n r)
        {"name": "svd_320x128", "kind": "svd", "p": 320, "q": 128, "keep": 64},
        # the same for the d = 100 chain at rank 256 and block 8
        {"name": "svd_2048x512", "kind": "svd", "p": 2048, "q": 512, "keep": 256},
        # a whole block eigensolve, chosen method
        {"name": "eigb_d12", "kind": "eigb", "d": 12, "rmax": 128, "block": 5, "start_rank": 16,
         "method": "split"},
        # two steps of the complex time stepper: d = 16, n = 32, rank 8
        {"name": "ksl_d16_n32", "kind": "ksl", "d": 16, "n": 32, "rank": 8, "steps": 2},
        # a whole linear solve on a grid
        {"name": "amen_d4_n24", "kind": "amen", "d": 4, "n": 24, "rank": 3},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: both ends, odd and ragged sizes."""
    kind = rng.choice(["apply", "apply", "apply", "split", "phi", "zapply", "qr", "svd", "eigb",
                       "ksl", "amen"])
    if kind in ("apply", "split"):
        method = "plain" if kind == "apply" else "split"
        if rng.random() < 0.6:
            r1 = _logint(rng, 8, 256)
            r2 = max(4, min(256, int(r1 * rng.uniform(0.6, 1.4))))
            return {"kind": "apply", "op": "chain", "method": method, "r1": r1, "n": 2, "r2": r2,
                    "nvec": rng.randint(1, 8)}
        r1 = _logint(rng, 4, 100)
        r2 = max(3, min(100, int(r1 * rng.uniform(0.6, 1.4))))
        return {"kind": "apply", "op": "grid", "method": method, "r1": r1,
                "n": rng.randint(16, 64), "r2": r2, "nvec": rng.randint(1, 4)}
    if kind == "phi":
        if rng.random() < 0.5:
            r1 = _logint(rng, 8, 256)
            return {"kind": "phi", "op": "chain", "r1": r1, "n": 2,
                    "r2": max(4, min(256, int(r1 * rng.uniform(0.6, 1.4))))}
        r1 = _logint(rng, 4, 100)
        return {"kind": "phi", "op": "grid", "r1": r1, "n": rng.randint(16, 64),
                "r2": max(3, min(100, int(r1 * rng.uniform(0.6, 1.4))))}
    if kind == "zapply":
        r1 = _logint(rng, 4, 64)
        return {"kind": "zapply", "r1": r1, "n": rng.randint(8, 32),
                "r2": max(3, min(64, int(r1 * rng.uniform(0.6, 1.4)))),
                "nvec": rng.choice([1, 1, 2, 4])}
    if kind == "qr":
        cols = _logint(rng, 8, 128)
        return {"kind": "qr", "rows": cols * rng.randint(2, 64) - rng.randint(0, cols - 1),
                "cols": cols}
    if kind == "svd":
        q = _logint(rng, 16, 400)
        return {"kind": "svd", "p": int(q * rng.uniform(1.0, 4.0)), "q": q, "keep": (q + 1) // 2}
    if kind == "eigb":
        d = rng.randint(8, 11)
        return {"kind": "eigb", "d": d, "rmax": 2 ** ((d + 1) // 2 + 1), "block": rng.randint(2, 5),
                "start_rank": rng.randint(6, 16), "method": rng.choice(["split", "plain"])}
    if kind == "ksl":
        return {"kind": "ksl", "d": rng.randint(4, 16), "n": rng.randint(12, 32),
                "rank": rng.randint(4, 10), "steps": 1}
    return {"kind": "amen", "d": 4, "n": rng.randint(12, 22), "rank": rng.randint(2, 3)}


# ------------------------------------------------------------------ the inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _znormal(g, *shape):
    return torch.complex(_normal(g, *shape), _normal(g, *shape)) * math.sqrt(0.5)


def _core(ra, n, m, packed, k):
    off = sum(ra[i] * n[i] * m[i] * ra[i + 1] for i in range(k))
    return np.asarray(packed[off:off + ra[k] * n[k] * m[k] * ra[k + 1]])


def _op_core(op, n, seed):
    """An interior operator core (ra1, n, n, ra2), flat, and its rank."""
    if op == "chain":
        n_, m_, ra, packed = operators.xxz_mpo(6, delta=0.5 + (seed % 1000) / 1000.0)
    elif op == "grid":
        n_, m_, ra, packed = operators.amen_operator(d=4, n=n, sigma_frac=0.2 + (seed % 100) / 500.0)
        return _core(ra, n_, m_, packed, 1), ra[1]
    else:
        n_, m_, ra, packed = operators.ksl_operator(d=4, n=n, rank=4, seed=seed)
        return _core(ra, n_, m_, packed, 1), ra[1]
    return _core(ra, n_, m_, packed, 2), ra[2]


def _local_inputs(case, seed):
    g = _gen(seed)
    r1, n, r2 = case["r1"], case["n"], case["r2"]
    core, ra = _op_core(case["op"], n, seed)
    nv = case.get("nvec", 1)
    return {"ra": ra, "A": torch.from_numpy(core).to(DEV),
            "phi1": _normal(g, r1 * r1 * ra) / math.sqrt(r1),
            "phi2": _normal(g, r2 * ra * r2) / math.sqrt(r2),
            "x": _normal(g, nv * r1 * n * r2) / math.sqrt(r1 * n * r2),
            "y": _normal(g, nv * r1 * n * r2) / math.sqrt(r1 * n * r2)}


def _z_inputs(case, seed):
    g = _gen(seed)
    r1, n, r2, nv = case["r1"], case["n"], case["r2"], case["nvec"]
    core, ra = _op_core("ksl", n, seed)
    return {"ra": ra, "A": torch.from_numpy(core).to(DEV).to(torch.complex128),
            "phi1": _znormal(g, r1 * r1 * ra) / math.sqrt(r1),
            "phi2": _znormal(g, r2 * ra * r2) / math.sqrt(r2),
            "x": _znormal(g, nv * r1 * n * r2) / math.sqrt(r1 * n * r2),
            "xt": _znormal(g, nv * r1 * n * r2) / math.sqrt(r1 * n * r2)}


def _svd_block(case, seed):
    """p x q (column-major, flat) with singular values over thirteen decades,
    as the local blocks of a converging sweep have them."""
    g = _gen(seed)
    p, q = case["p"], case["q"]
    r = min(p, q)
    U, V = (torch.from_numpy(np.linalg.qr(_normal(g, k, r).cpu().numpy())[0]).to(DEV)
            for k in (p, q))
    step = torch.rand(r, generator=g, device=DEV, dtype=torch.float64) + 0.5
    e = torch.cumsum(step, 0)
    s = 10.0 ** (-13.0 * e / e[-1])
    return ((U * s) @ V.T).T.contiguous().reshape(-1)


def _eigb_inputs(case, seed):
    d = case["d"]
    delta = 0.8 + 0.4 * ((seed * 2654435761) % 1000) / 1000.0
    n, m, ra, crA = operators.xxz_mpo(d, delta=delta)
    _, ry, y = operators.random_tt(d, 2, case["start_rank"], last=case["block"], seed=seed)
    return delta, n, m, ra, crA, ry, y


def _ksl_inputs(case, seed):
    d, n = case["d"], case["n"]
    n_, m_, ra, crA = operators.ksl_operator(d=d, n=n, rank=4, seed=seed)
    _, ry, y = operators.random_tt_complex(d, n, case["rank"], seed=seed + 1)
    nrm = operators.tt_norm(d, n, ry, y)
    scale = nrm ** (-1.0 / d)   # spread over the cores
    return n_, m_, ra, crA, ry, y * scale


def _amen_inputs(case, seed):
    d, n = case["d"], case["n"]
    n_, m_, ra, crA = operators.amen_operator(d=d, n=n)
    _, ry, y = operators.random_tt(d, n, case["rank"], seed=seed)
    _, rx, x0 = operators.random_tt(d, n, 2, seed=seed + 1)
    return n_, m_, ra, crA, ry, y, rx, x0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "apply":
        s = _local_inputs(case, seed)
        r1, n, r2, nv = case["r1"], case["n"], case["r2"], case["nvec"]
        s["op"] = ttgpu.LocalOp(r1, n, r2, r1, n, r2, s["ra"], s["ra"], s["phi1"], s["A"],
                                s["phi2"], nvec_max=nv, method=case["method"])
        s["out"] = torch.empty_like(s["x"])
    elif kind == "phi":
        s = _local_inputs(case, seed)
        s["left"] = torch.empty(case["r2"] ** 2 * s["ra"], device=DEV, dtype=torch.float64)
        s["right"] = torch.empty(case["r1"] ** 2 * s["ra"], device=DEV, dtype=torch.float64)
    elif kind == "zapply":
        s = _z_inputs(case, seed)
        s["out"], s["outt"] = torch.empty_like(s["x"]), torch.empty_like(s["xt"])
    elif kind == "qr":
        rows, cols = case["rows"], case["cols"]
        s = {"core": _normal(_gen(seed), rows * cols)}
        s["q"] = torch.empty_like(s["core"])
        s["r"] = torch.empty(min(rows, cols) * cols, device=DEV, dtype=torch.float64)
    elif kind == "svd":
        p, q = case["p"], case["q"]
        r = min(p, q)
        s = {"block": _svd_block(case, seed)}
        s["u"] = torch.empty(p * r, device=DEV, dtype=torch.float64)
        s["s"] = torch.empty(r, device=DEV, dtype=torch.float64)
        s["vt"] = torch.empty(r * q, device=DEV, dtype=torch.float64)
    elif kind == "eigb":
        delta, n, m, ra, crA, ry, y = _eigb_inputs(case, seed)
        s = {"n": n, "m": m, "ra": ra, "crA": crA, "ry": ry, "y": y, "ctx": _driver_ctx()}
    elif kind == "ksl":
        n, m, ra, crA, ry, y = _ksl_inputs(case, seed)
        s = {"n": n, "m": m, "ra": ra, "crA": crA, "ry": ry, "y": y, "ctx": _driver_ctx()}
    elif kind == "amen":
        n, m, ra, crA, ry, y, rx, x0 = _amen_inputs(case, seed)
        s = {"n": n, "m": m, "ra": ra, "crA": crA, "ry": ry, "y": y, "rx": rx, "x0": x0,
             "ctx": _driver_ctx()}
    else:
        raise ValueError(kind)
    s["case"] = case
    return s


def _full(n, r, cores):
    """The tensor of a TT vector, flat with the first index fastest."""
    T = np.ones((1, 1))
    off = 0
    for k in range(len(n)):
        sz = r[k] * n[k] * r[k + 1]
        c = cores[off:off + sz].reshape(r[k], n[k] * r[k + 1], order="F")
        off += sz
        T = (T @ c).reshape(-1, r[k + 1], order="F")
    return T[:, 0]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "apply":
        s["op"].apply(s["x"], s["out"], case["nvec"])
        return s["out"]
    if kind == "phi":
        r1, n, r2, ra = case["r1"], case["n"], case["r2"], s["ra"]
        ttgpu.phi_left(r1, n, r2, r1, n, r2, ra, ra, s["phi1"], s["A"], s["x"], s["y"], s["left"])
        ttgpu.phi_right(r1, n, r2, r1, n, r2, ra, ra, s["phi2"], s["A"], s["x"], s["y"], s["right"])
        return {"left": s["left"], "right": s["right"]}
    if kind == "zapply":
        r1, n, r2, ra, nv = case["r1"], case["n"], case["r2"], s["ra"], case["nvec"]
        ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, s["phi1"], s["A"], s["phi2"], s["x"], s["out"], nv)
        ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, s["phi1"], s["A"], s["phi2"], s["xt"], s["outt"],
                     nv, transp=True)
        return {"y": s["out"], "yt": s["outt"]}
    if kind == "qr":
        s["q"].copy_(s["core"])     # dqr works in place; the sweep keeps its core
        ttgpu.dqr(case["rows"], case["cols"], s["q"], s["r"])
        return {"q": s["q"], "r": s["r"]}
    if kind == "svd":
        p, q, k = case["p"], case["q"], case["keep"]
        r = min(p, q)
        ttgpu.dgesvd(p, q, s["block"], s["u"], s["s"], s["vt"])
        # what a sweep goes on with: the singular values and the block
        # truncated to its rank cap.  The signs of single singular vectors
        # are free, so the factors are multiplied out as the sweep does.
        u = s["u"].view(r, p)[:k]                  # rows: left vectors
        vt = s["vt"].view(q, r)[:, :k]
        return {"s": s["s"], "block": vt @ (u * s["s"][:k, None])}   # (q, p)
    if kind == "eigb":
        # eigenvectors of a multiplet and the gauge of the cores are free:
        # the eigenvalues are what the call determines
        lam, _, _ = ttgpu.tt_eigb(case["d"], s["n"], s["m"], s["ra"], s["crA"], s["y"], s["ry"],
                                  1e-8, case["rmax"], case["block"], max_full_size=200,
                                  method=case["method"], ctx=s["ctx"])
        return lam
    if kind == "ksl":
        cores, _ = ttgpu.ztt_ksl(case["d"], s["n"], s["m"], s["ra"], s["crA"], s["y"], s["ry"], 1e-3,
                                 64, nsteps=case["steps"], ctx=s["ctx"])
        return cores
    cores, rx = ttgpu.dtt_amen_solve(case["d"], s["n"], s["m"], s["ry"], s["ra"], s["crA"], s["y"],
                                     s["x0"], s["rx"], 1e-8, ctx=s["ctx"])
    return _full(s["n"], rx, cores)   # the solution; its cores' gauge is free


# ------------------------------------------------------- what a pass cannot avoid
def _bfun_flops(r1, n, r2, ra):
    return 2.0 * (r1 * n * r2 * ra * r2 + ra * n * n * ra * r2 * r1 + r1 * n * r2 * r1 * ra)


def _qr_flops(p, q):
    r = min(p, q)
    return 4.0 * p * q * r - 4.0 * r * r * r / 3.0 if p >= q else 4.0 * p * p * q


def _rank(case):
    return {"chain": 5, "grid": 3}[case["op"]]


def work(case):
    kind = case["kind"]
    if kind in ("apply", "phi"):
        r1, n, r2, ra, nv = case["r1"], case["n"], case["r2"], _rank(case), case.get("nvec", 1)
        f = _bfun_flops(r1, n, r2, ra) * nv
        b = 8.0 * (r1 * r1 * ra + r2 * r2 * ra + ra * n * n * ra + 2 * nv * r1 * n * r2)
        if kind == "phi":     # two updates, each with old and new interface
            return {"bytes": 2 * b, "flops": 2 * f}
        return {"bytes": b, "flops": f}
    if kind == "zapply":
        r1, n, r2, ra, nv = case["r1"], case["n"], case["r2"], 6, case["nvec"]
        b = 16.0 * (r1 * r1 * ra + r2 * r2 * ra + ra * n * n * ra + 4 * nv * r1 * n * r2)
        return {"bytes": b, "flops": 8.0 * _bfun_flops(r1, n, r2, ra) * nv}
    if kind == "qr":
        rows, cols = case["rows"], case["cols"]
        return {"bytes": 8.0 * (2 * rows * cols + cols * cols), "flops": _qr_flops(rows, cols)}
    if kind == "svd":
        p, q = case["p"], case["q"]
        return {"bytes": 8.0 * (2 * p * q + q * q),
                "flops": _qr_flops(p, q) + 20.0 * q ** 3 + 2.0 * p * q * case["keep"]}
    # whole calls: operator, start and result once; per core and half sweep
    # one block product, one factorisation and one interface update
    if kind == "eigb":
        d, B = case["d"], case["block"]
        r = [min(case["rmax"], 2 ** k, 2 ** (d - k)) for k in range(d + 1)]
        f = 4 * sum(_bfun_flops(r[k], 2, r[k + 1], 5) * (B + 1) + 26.0 * B * r[k] * (2 * r[k + 1]) ** 2
                    for k in range(d))
        return {"bytes": 8.0 * (d * 100 + 2 * B * sum(r[k] * 2 * r[k + 1] for k in range(d))),
                "flops": f}
    d, n = case["d"], case["n"]
    if kind == "ksl":
        r, steps = case["rank"], case["steps"]
        f = 4.0 * steps * 2 * d * (10 * _bfun_flops(r, n, r, 6) + _qr_flops(r * n, r))
        return {"bytes": 16.0 * (d * 36 * n * n + 2 * d * r * n * r), "flops": f}
    r = 5 * case["rank"]
    f = 2.0 * d * (10 * _bfun_flops(r, n, r, 3) + _qr_flops(r * n, r))
    return {"bytes": 8.0 * (d * 9 * n * n + d * r * n * r + n ** d), "flops": f}


# ---------------------------------------------------------------- 64-bit values
def _views(case, s):
    """phi1[a1,b1,c1], A[a2,j,i,a1], phi2[c2,a2,b2], x[v,b2,j,b1]: the flat
    column-major arrays as row-major views."""
    r1, n, r2, ra = case["r1"], case["n"], case["r2"], s["ra"]
    return (s["phi1"].view(ra, r1, r1), s["A"].view(ra, n, n, ra), s["phi2"].view(r2, ra, r2))


def _apply_exact(p1, A, p2, x):
    # y[v,c2,i,c1] = phi1[a1,b1,c1] A[a2,j,i,a1] phi2[c2,a2,b2] x[v,b2,j,b1]
    t = torch.einsum("cae,vejb->vcajb", p2, x)
    t = torch.einsum("ajid,vcajb->vcidb", A, t)
    return torch.einsum("dbz,vcidb->vciz", p1, t)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("apply", "phi"):
        s = _local_inputs(case, seed)
        r1, n, r2, nv = case["r1"], case["n"], case["r2"], case.get("nvec", 1)
        p1, A, p2 = _views(case, s)
        x, y = s["x"].view(nv, r2, n, r1), s["y"].view(nv, r2, n, r1)
        if kind == "apply":
            return _apply_exact(p1, A, p2, x).reshape(-1)
        # left[a2,b2,c2] = phi1[a1,b1,c1] y[c2,i,c1] A[a2,j,i,a1] x[b2,j,b1]
        t = torch.einsum("dbz,ciz->cidb", p1, y[0])
        t = torch.einsum("ajid,cidb->cajb", A, t)
        left = torch.einsum("cajb,ejb->aec", t, x[0])
        # right[c1,a1,b1] = x[b2,j,b1] phi2[c2,a2,b2] A[a2,j,i,a1] y[c2,i,c1]
        t = torch.einsum("cae,ejb->cajb", p2, x[0])
        t = torch.einsum("ajid,cajb->cidb", A, t)
        right = torch.einsum("cidb,ciz->zdb", t, y[0])
        return {"left": left.reshape(-1), "right": right.reshape(-1)}
    if kind == "zapply":
        s = _z_inputs(case, seed)
        r1, n, r2, nv = case["r1"], case["n"], case["r2"], case["nvec"]
        p1, A, p2 = _views(case, s)
        y = _apply_exact(p1, A, p2, s["x"].view(nv, r2, n, r1))
        t = torch.einsum("dbz,vciz->vcidb", p1.conj(), s["xt"].view(nv, r2, n, r1))
        t = torch.einsum("ajid,vcidb->vcajb", A.conj(), t)
        yt = torch.einsum("cae,vcajb->vejb", p2.conj(), t)
        return {"y": y.reshape(-1), "yt": yt.reshape(-1)}
    if kind == "qr":
        rows, cols = case["rows"], case["cols"]
        a = _normal(_gen(seed), rows * cols).cpu().numpy().reshape(rows, cols, order="F")
        q, r = np.linalg.qr(a)
        return {"q": q.ravel(order="F"), "r": r.ravel(order="F")}
    if kind == "svd":
        p, q, k = case["p"], case["q"], case["keep"]
        m = _svd_block(case, seed).view(q, p).T.cpu().numpy()
        u, s, vt = np.linalg.svd(m, full_matrices=False)
        return {"s": s, "block": ((u[:, :k] * s[:k]) @ vt[:k]).T.copy()}
    if kind == "eigb":
        # the total spin along z is conserved: one dense block per value of it
        d = case["d"]
        delta = _eigb_inputs(case, seed)[0]
        idx = np.arange(2 ** d)
        ups = sum((idx >> k) & 1 for k in range(d))
        vals = []
        for up in range(d + 1):
            st = idx[ups == up]
            H = np.zeros((len(st), len(st)))
            for k in range(d - 1):
                same = ((st >> k) & 1) == ((st >> (k + 1)) & 1)
                H[np.arange(len(st)), np.arange(len(st))] += np.where(same, 0.25, -0.25) * delta
                col = np.nonzero(~same)[0]
                H[np.searchsorted(st, st[col] ^ (3 << k)), col] += 0.5
            vals.append(np.linalg.eigvalsh(H))
        return np.sort(np.concatenate(vals))[:case["block"]]
    if kind == "amen":
        n_, m_, ra, crA, ry, y, rx, x0 = _amen_inputs(case, seed)
        d, n = case["d"], case["n"]
        lap = 2 * torch.eye(n, dtype=torch.float64) - torch.diag(torch.ones(n - 1, dtype=torch.float64), 1) \
            - torch.diag(torch.ones(n - 1, dtype=torch.float64), -1)
        lap = lap.to(DEV)
        grid = torch.arange(n, dtype=torch.float64, device=DEV)
        gauss = torch.exp(-((grid - (n - 1) / 2.0) ** 2) / (0.3 * n) ** 2)
        pot = gauss
        for _ in range(d - 1):
            pot = pot.unsqueeze(-1) * gauss
        b = torch.from_numpy(_full(n_, ry, y)).to(DEV).view(*([n] * d))

        def mul(v):
            out = pot * v
            for k in range(d):
                out = out + torch.movedim(torch.tensordot(lap, v, dims=([1], [k])), 0, k)
            return out

        x = torch.zeros_like(b)
        r = b.clone()
        p = r.clone()
        rr = (r * r).sum()
        for _ in range(600):     # conjugate gradients to rounding
            q = mul(p)
            a = rr / (p * q).sum()
            x = x + a * p
            r = r - a * q
            new = (r * r).sum()
            p = r + (new / rr) * p
            rr = new
            if float(new) <= 1e-32 * float((b * b).sum()):
                break
        return x.reshape(-1).cpu().numpy()
    return None   # ksl: a splitting scheme; its result is its own definition
