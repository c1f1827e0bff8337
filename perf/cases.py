"""The work that users of the library have it do, as cases that can be timed and compared.

A case is a dict of plain values; its ``kind`` names the call:

* ``potrf``, ``posv``: uniform batches through ``blast_gb300.blast`` (a batch of one is BLAST's own call)
* ``gemm``, ``trsm``, ``riccati``: the uniform BLAS-3 calls, with BLAST's transposed views
* ``posv_ragged``, ``posv_mixed``: ragged Cholesky solves through ``PosvPlan``, in binary64 and in mixed
  precision with refinement
* ``lu_ragged``, ``lu_mixed``: ragged LU solves through ``GesvPlan`` and ``MixedGesvPlan``
* ``spd_grad``: the differentiable ragged solve, forward and backward
* ``host``: a batch in pinned host memory through ``PosvHostPipeline``

``prepare`` makes the inputs on the GPU from the seed alone and the plan that a program keeps, ``run`` is one pass
through the public entry points, ``exact`` is the same result by torch in binary64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from blast_gb300 import blast
from blast_gb300.autograd import spd_solve_packed
from blast_gb300.host import PosvHostPipeline, pinned_col_major
from blast_gb300.ragged import GesvPlan, MixedGesvPlan, Packed, PosvPlan

F64 = torch.float64


def listed():
    return [
        # one small factorisation, as a controller calls BLAST inside its loop: launch and call latency
        {"name": "potrf_one_24", "kind": "potrf", "n": 24, "batch": 1},
        # the small-matrix gemm batch of BLAST's benchmarks
        {"name": "gemm_24", "kind": "gemm", "m": 24, "n": 24, "k": 24, "batch": 10_000, "ta": False, "tb": False,
         "alpha": 1.0, "beta": 1.0},
        # odd sizes, a transposed view, padded columns and scalars other than one
        {"name": "gemm_odd_trans", "kind": "gemm", "m": 57, "n": 39, "k": 23, "batch": 3_000, "ta": False, "tb": True,
         "alpha": -1.0, "beta": 0.5},
        # the batched Cholesky solve of the benchmark
        {"name": "posv_48", "kind": "posv", "n": 48, "nrhs": 8, "batch": 50_000},
        # triangular solves with several right-hand sides against a transposed factor
        {"name": "trsm_64", "kind": "trsm", "m": 64, "n": 16, "batch": 2_000, "upper": True, "unit": False,
         "trans": True},
        # the Riccati step, chol(C + A^T A)
        {"name": "riccati_60", "kind": "riccati", "n": 60, "k": 30, "batch": 20_000},
        # ragged Cholesky solves in binary64, then in mixed precision with refinement
        {"name": "posv_ragged_512", "kind": "posv_ragged", "lo": 64, "hi": 512, "nrhs": 1, "count": 2_048},
        {"name": "posv_mixed_512", "kind": "posv_mixed", "lo": 64, "hi": 512, "nrhs": 1, "count": 2_048},
        # ragged general systems, sizes spread over their logarithm
        {"name": "lu_ragged_256", "kind": "lu_ragged", "lo": 4, "hi": 256, "nrhs": 1, "count": 8_000},
        {"name": "lu_mixed_256", "kind": "lu_mixed", "lo": 4, "hi": 256, "nrhs": 1, "count": 8_000},
        # a layer that solves SPD systems inside a differentiable program: forward and backward
        {"name": "spd_grad_128", "kind": "spd_grad", "lo": 32, "hi": 128, "nrhs": 1, "count": 4_096, "keep": True},
        # a batch that lives in host memory, there and back
        {"name": "host_48", "kind": "host", "n": 48, "nrhs": 8, "batch": 10_000},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    kind = rng.choice(["potrf", "gemm", "gemm", "posv", "posv", "trsm", "riccati", "posv_ragged", "posv_ragged",
                       "posv_mixed", "lu_ragged", "lu_mixed", "spd_grad", "host"])
    if kind == "gemm":
        c = {"kind": kind, "m": _log_int(rng, 1, 128), "n": _log_int(rng, 1, 128), "k": _log_int(rng, 1, 128),
             "ta": rng.random() < 0.5, "tb": rng.random() < 0.5, "alpha": rng.choice([1.0, -1.0, 0.75]),
             "beta": rng.choice([0.0, 1.0, -0.5])}
        most, per = 30_000, c["m"] * c["n"] * c["k"] + 50 * (c["m"] + c["n"] + c["k"])
    elif kind == "trsm":
        c = {"kind": kind, "m": _log_int(rng, 2, 128), "n": _log_int(rng, 1, 64), "upper": rng.random() < 0.5,
             "unit": rng.random() < 0.3, "trans": rng.random() < 0.5}
        most, per = 10_000, c["m"] * c["m"] * (c["n"] + 8)
    elif kind == "riccati":
        c = {"kind": kind, "n": _log_int(rng, 4, 64), "k": _log_int(rng, 1, 64)}
        most, per = 20_000, c["n"] ** 2 * (c["n"] + c["k"])
    elif kind in ("potrf", "posv", "host"):
        c = {"kind": kind, "n": _log_int(rng, 2, 64 if kind == "host" else 256)}
        if kind != "potrf":
            c["nrhs"] = _log_int(rng, 1, 16)
        most = 10_000 if kind == "host" else 50_000
        per = c["n"] ** 3 + 4 * c["n"] ** 2 * c.get("nrhs", 1)
    else:
        lo, hi = {"spd_grad": (2, 128), "lu_ragged": (2, 256), "lu_mixed": (2, 256)}.get(kind, (8, 512))
        a, b = _log_int(rng, lo, hi), _log_int(rng, lo, hi)
        c = {"kind": kind, "lo": min(a, b), "hi": max(a, b), "nrhs": 1 if rng.random() < 0.7 else rng.randint(2, 4),
             "count": 0}
        if kind in ("posv_mixed", "lu_mixed"):
            c["nrhs"] = 1
        if kind == "spd_grad":
            c["keep"] = rng.random() < 0.7
        most, per = 4_096, c["hi"] ** 3
        c["count"] = min(_log_int(rng, 1, most), max(1, int(5e10 / per)))
        return c
    c["batch"] = min(_log_int(rng, 1, most), max(1, int(1.5e9 / per)))
    return c


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=F64)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=F64) * 2 - 1


def _col(t):
    """A column-major copy of (batch, rows, cols)."""
    return t.mT.contiguous().mT


def _gram(g, batch, n):
    """Symmetric positive definite G G^T + n I."""
    G = _randn(g, batch, n, n)
    A = torch.bmm(G, G.mT)
    A.diagonal(dim1=-2, dim2=-1).add_(float(n))
    return A


def _sizes(case):
    """The instances' sizes, the same for every seed."""
    lo, hi, count = case["lo"], case["hi"], case["count"]
    rng = np.random.default_rng([lo, hi, count])
    if case["kind"] in ("lu_ragged", "lu_mixed"):
        return np.exp(rng.uniform(np.log(lo), np.log(hi + 1), count)).astype(np.int64).clip(lo, hi)
    return rng.integers(lo, hi + 1, count)


def _chunks(ns):
    """Instances in chunks of at most 256 MB when padded to the largest size, in the caller's order."""
    step = max(1, (1 << 25) // int(ns.max()) ** 2)
    return [slice(i, min(i + step, len(ns))) for i in range(0, len(ns), step)]


def _masks(ns):
    """(count, max n) mask of the rows that an instance has, on the GPU."""
    t = torch.from_numpy(ns).cuda()
    return torch.arange(int(ns.max()), device="cuda")[None, :] < t[:, None]


def _pack(padded, rows, cols):
    """Padded (count, r, c) matrices as one buffer of column-major matrices back to back."""
    return padded.mT[cols[:, :, None] & rows[:, None, :]]


def _unpack(flat, rows, cols):
    """The inverse of _pack, zeros in the padding."""
    out = torch.zeros(cols.shape[0], cols.shape[1], rows.shape[1], device="cuda", dtype=F64)
    out[cols[:, :, None] & rows[:, None, :]] = flat
    return out.mT


def _rhs_mask(count, nrhs):
    return torch.ones(count, nrhs, dtype=torch.bool, device="cuda")


def _ragged_matrices(case, ns, g):
    """The packed matrices of a ragged case: Gaussian for LU; Q diag(lambda) Q^T with condition 1e2, 1e4 or 1e6 (Q a
    product of reflections, lambda log-spaced) for the Cholesky solves; G G^T + n I for the differentiable one."""
    parts = []
    for s in _chunks(ns):
        n = ns[s]
        rows = _masks(n)
        cnt, m = rows.shape
        pair = rows[:, :, None] & rows[:, None, :]
        if case["kind"] in ("lu_ragged", "lu_mixed"):
            A = _randn(g, cnt, m, m)
        elif case["kind"] == "spd_grad":
            G = _randn(g, cnt, m, m) * pair
            A = torch.bmm(G, G.mT)
            A.diagonal(dim1=-2, dim2=-1).add_(torch.from_numpy(n).cuda()[:, None].to(F64))
        else:
            size = torch.from_numpy(n).cuda()[:, None].to(F64)
            power = 2.0 * torch.randint(1, 4, (cnt, 1), generator=g, device="cuda")
            at = torch.arange(m, device="cuda")[None, :] / (size - 1).clamp(min=1)
            A = torch.diag_embed((10.0 ** (-power * at)) * rows)
            for _ in range(6):
                v = _randn(g, cnt, m) * rows
                v = (v / v.norm(dim=1, keepdim=True))[:, :, None]
                w = torch.bmm(A, v)
                w = 2 * (w - v * torch.bmm(v.mT, w))
                A -= torch.bmm(torch.cat((v, w), 2), torch.cat((w, v), 2).mT)
            A = (A + A.mT) / 2
        parts.append(_pack(A, rows, rows))
    return torch.cat(parts)


def _ragged_inputs(case, seed):
    ns, g = _sizes(case), _gen(seed)
    A = _ragged_matrices(case, ns, g)
    b = _randn(g, int(ns.sum()) * case["nrhs"])
    return ns, A, b, g


def _uniform_inputs(case, seed):
    g = _gen(seed)
    kind, batch = case["kind"], case["batch"]
    if kind in ("potrf", "posv", "host"):
        A = _gram(g, batch, case["n"])
        return A, _randn(g, batch, case["n"], case["nrhs"]) if "nrhs" in case else None
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return _uniform(g, batch, m, k), _uniform(g, batch, k, n), _uniform(g, batch, m, n)
    if kind == "trsm":
        m = case["m"]
        A = _randn(g, batch, m, m) / math.sqrt(m)
        A.diagonal(dim1=-2, dim2=-1).copy_(1 + torch.rand(batch, m, generator=g, device="cuda", dtype=F64))
        return A, _randn(g, batch, m, case["n"])
    n, k = case["n"], case["k"]
    G = _uniform(g, batch, n, n)
    C = torch.bmm(G, G.mT)
    C.diagonal(dim1=-2, dim2=-1).add_(float(n))
    return _uniform(g, batch, k, n), C


def _storage(t, row_major):
    return t.contiguous() if row_major else _col(t)


def prepare(case, seed):
    kind = case["kind"]
    if "lo" in case:
        ns, A0, b0, g = _ragged_inputs(case, seed)
        rs = np.full_like(ns, case["nrhs"])
        if kind == "spd_grad":
            t = _randn(g, b0.numel())
            return {"case": case, "A": A0.requires_grad_(), "b": b0.requires_grad_(), "t": t, "ns": ns, "rs": rs}
        A, B = Packed(ns, ns, "cuda"), Packed(ns, rs, "cuda")
        A.buf.copy_(A0)
        B.buf.copy_(b0)
        if kind in ("lu_ragged", "lu_mixed"):  # solved in place: the systems of a pass arrive in A0, b0
            plan = GesvPlan(A, B) if kind == "lu_ragged" else MixedGesvPlan(A, B)
            return {"case": case, "plan": plan, "A": A, "B": B, "A0": A0, "b0": b0}
        X = Packed(ns, rs, "cuda")
        L = None if kind == "posv_mixed" else Packed(ns, ns, "cuda")
        return {"case": case, "plan": PosvPlan(A, B, X, L, mixed=L is None), "X": X, "L": L}
    data = _uniform_inputs(case, seed)
    batch = case["batch"]
    if kind in ("potrf", "posv"):
        A, B = data
        s = {"case": case, "A": _col(A), "L": blast.col_major((batch,), case["n"], case["n"]).zero_()}
        if B is not None:
            s |= {"B": _col(B), "X": blast.col_major((batch,), case["n"], case["nrhs"])}
        return s
    if kind == "host":
        n, r = case["n"], case["nrhs"]
        hA, hB = pinned_col_major(batch, n, n), pinned_col_major(batch, n, r)
        hA.copy_(data[0])
        hB.copy_(data[1])
        hL, hX = pinned_col_major(batch, n, n).zero_(), pinned_col_major(batch, n, r)
        return {"case": case, "pipe": PosvHostPipeline(n, r, batch, "cuda", transport="mirror"), "A": hA, "B": hB,
                "L": hL, "X": hX, "info": torch.zeros(batch, dtype=torch.int32).pin_memory()}
    if kind == "gemm":
        A, B, C = data
        m, n = case["m"], case["n"]
        return {"case": case, "A": _storage(A, case["ta"]), "B": _storage(B, case["tb"]), "C": _col(C),
                "D": blast.col_major((batch,), m, n)}
    if kind == "trsm":
        A, B = data
        return {"case": case, "A": _storage(A, case["trans"]), "B": _col(B),
                "X": blast.col_major((batch,), case["m"], case["n"])}
    A, C = data  # A is k x n column-major; the call takes its transposed view
    return {"case": case, "A": _col(A).mT, "C": _col(C), "D": blast.col_major((batch,), case["n"], case["n"]).zero_()}


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "potrf":
        return {"info": blast.potrf(s["A"], s["L"]), "L": s["L"]}
    if kind == "posv":
        return {"info": blast.posv(s["A"], s["L"], s["B"], s["X"]), "L": s["L"], "X": s["X"]}
    if kind == "gemm":
        return blast.gemm(case["alpha"], s["A"], s["B"], case["beta"], s["C"], s["D"])
    if kind == "trsm":
        return blast.trsm(blast.UPPER if case["upper"] else blast.LOWER, case["unit"], s["A"], s["B"], s["X"])
    if kind == "riccati":
        return {"info": blast.syrk_potrf(1.0, s["A"], 1.0, s["C"], s["D"]), "D": s["D"]}
    if kind == "posv_ragged":
        s["plan"].run()
        return {"info": s["plan"].info, "L": s["L"].buf, "X": s["X"].buf}
    if kind == "posv_mixed":
        s["plan"].run()
        return {"info": s["plan"].info, "X": s["X"].buf}
    if kind in ("lu_ragged", "lu_mixed"):
        s["B"].buf.copy_(s["b0"])
        if kind == "lu_ragged":
            s["A"].buf.copy_(s["A0"])
        s["plan"].run()
        out = {"info": s["plan"].info, "ipiv": s["plan"].ipiv.buf, "X": s["B"].buf}
        return out | {"LU": s["A"].buf} if kind == "lu_ragged" else out
    if kind == "spd_grad":
        x = spd_solve_packed(s["A"], s["b"], s["ns"], s["rs"], keep_factor=case["keep"])
        gA, gb = torch.autograd.grad(0.5 * ((x - s["t"]) ** 2).sum(), (s["A"], s["b"]))
        return {"x": x.detach(), "gA": gA, "gb": gb}
    s["pipe"].run(s["A"], s["B"], s["L"], s["X"], s["info"])
    return {"info": s["info"], "L": s["L"], "X": s["X"]}


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _solve_flops(n, r):
    return n ** 3 / 3 + n ** 2 / 2 + n / 6 + 2.0 * n * n * r


def work(case):
    kind = case["kind"]
    if "lo" in case:
        ns, r = _sizes(case).astype(np.float64), case["nrhs"]
        tri, sq, vec = 8 * (ns * (ns + 1) / 2).sum(), 8 * (ns ** 2).sum(), 8 * ns.sum() * r
        chol, lu = _solve_flops(ns, r).sum(), (2 * ns ** 3 / 3 - ns ** 2 / 2 + 5 * ns / 6 + 2 * ns ** 2 * r).sum()
        if kind == "posv_ragged":
            return {"bytes": 2 * tri + 2 * vec, "flops": chol}
        if kind == "posv_mixed":
            return {"bytes": tri + 2 * vec, "flops": chol}
        if kind == "spd_grad":  # forward reads lower(A), b, writes x; backward writes both gradients
            return {"bytes": tri + sq + 4 * vec, "flops": chol + (4 * ns ** 2 * r).sum()}
        return {"bytes": (2 if kind == "lu_ragged" else 1) * sq + 2 * vec + 4 * ns.sum(), "flops": lu}
    b = case["batch"]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * b * (m * k + k * n + 2 * m * n), "flops": 2 * b * m * n * k}
    if kind == "trsm":
        m, n = case["m"], case["n"]
        return {"bytes": 8 * b * (m * (m + 1) / 2 + 2 * m * n), "flops": b * m * m * n}
    n = case["n"]
    tri = n * (n + 1) / 2
    if kind == "riccati":
        return {"bytes": 8 * b * (2 * tri + n * case["k"]), "flops": b * (n * (n + 1) * case["k"] + n ** 3 / 3)}
    r = case.get("nrhs", 0)
    return {"bytes": 8 * b * (2 * tri + 2 * n * r) + 4 * b, "flops": b * _solve_flops(n, r)}


# ---------------------------------------------------------------------------------------------
# The same results by torch in binary64
# ---------------------------------------------------------------------------------------------
def _exact_ragged(case, seed):
    ns, A, b, g = _ragged_inputs(case, seed)
    kind, r = case["kind"], case["nrhs"]
    t = _randn(g, b.numel()) if kind == "spd_grad" else None
    sq = np.concatenate([[0], np.cumsum(ns * ns)])
    vec = np.concatenate([[0], np.cumsum(ns * r)])
    out = {}
    for s in _chunks(ns):
        lo, hi = s.start, s.stop
        rows, cols = _masks(ns[s]), _rhs_mask(hi - lo, r)
        M = _unpack(A[sq[lo]:sq[hi]], rows, rows)
        M = M + torch.diag_embed((~rows).to(F64))
        B = _unpack(b[vec[lo]:vec[hi]], rows, cols)
        if kind in ("lu_ragged", "lu_mixed"):
            LU, piv = torch.linalg.lu_factor(M)
            got = {"X": _pack(torch.linalg.lu_solve(LU, piv, B), rows, cols)}
            if kind == "lu_ragged":
                got["LU"] = _pack(LU, rows, rows)
        else:
            L = torch.linalg.cholesky(M)
            X = torch.cholesky_solve(B, L)
            if kind == "spd_grad":
                T = _unpack(t[vec[lo]:vec[hi]], rows, cols)
                Bb = torch.cholesky_solve(X - T, L)
                S = torch.bmm(Bb, X.mT)
                got = {"x": _pack(X, rows, cols), "gb": _pack(Bb, rows, cols), "gA": _pack(-(S + S.mT) / 2, rows, rows)}
            else:
                got = {"X": _pack(X, rows, cols)}
                if kind == "posv_ragged":
                    got["L"] = _pack(L, rows, rows)
        for k, v in got.items():
            out.setdefault(k, []).append(v)
    return {k: torch.cat(v) for k, v in out.items()}


def exact(case, seed):
    kind = case["kind"]
    if "lo" in case:
        out = _exact_ragged(case, seed)
        keys = {"posv_ragged": ("info",), "posv_mixed": ("info",), "spd_grad": ()}.get(kind, ("info", "ipiv"))
        return {**out, **{k: None for k in keys}}
    data = _uniform_inputs(case, seed)
    if kind == "gemm":
        A, B, C = data
        return case["alpha"] * torch.bmm(A, B) + case["beta"] * C
    if kind == "trsm":
        A, B = data
        return torch.linalg.solve_triangular(A, B, upper=case["upper"], unitriangular=case["unit"])
    if kind == "riccati":
        A, C = data
        return {"info": None, "D": torch.linalg.cholesky(C + torch.bmm(A.mT, A))}
    A, B = data
    L = torch.linalg.cholesky(A)
    out = {"info": None, "L": L}
    if B is not None:
        out["X"] = torch.cholesky_solve(B, L)
    return {k: v.cpu() if v is not None and kind == "host" else v for k, v in out.items()}
