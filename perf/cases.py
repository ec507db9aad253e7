"""Workloads of the library's public entry points, with inputs made from a seed.

Every matrix is uniform noise on [-0.5, 0.5] plus sqrt(n)/2 on a randomly
row-permuted diagonal: well conditioned at every order (so that solutions can be
compared digit by digit), while partial pivoting interchanges a row at nearly
every column, as it does on general dense matrices. Matrices are column-major
(a torch tensor holds the transpose), as the entry points take them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import scalapack_gb300 as sl

F64 = torch.float64


def listed():
    return [
        # a solve inside somebody's inner loop: latency and launches
        {"name": "gesv_n17", "kind": "gesv", "n": 17, "nrhs": 1, "nb": 0},
        # a small dense system with a small distribution block (the smoke test's size)
        {"name": "gesv_n600", "kind": "gesv", "n": 600, "nrhs": 2, "nb": 64},
        # an ordinary dense solve
        {"name": "gesv_n4096", "kind": "gesv", "n": 4096, "nrhs": 16, "nb": 256},
        # the benchmark's configuration: the large dense solve
        {"name": "gesv_n16384", "kind": "gesv", "n": 16384, "nrhs": 16, "nb": 256},
        # factors of a ragged tall matrix
        {"name": "getrf_6001x3007", "kind": "getrf", "m": 6001, "n": 3007, "nb": 256},
        # factored once, solved for one vector after another
        {"name": "getrs_n8192_r1", "kind": "getrs", "n": 8192, "nrhs": 1, "trans": "N"},
        # the transposed system (adjoints, condition estimates), a block of vectors
        {"name": "getrst_n8192_r16", "kind": "getrs", "n": 8192, "nrhs": 16, "trans": "T"},
        # the Fortran-style call on ordinary host arrays, copies included
        {"name": "pdgesv_n2000", "kind": "pdgesv", "n": 2000, "nrhs": 1, "nb": 64},
        # thousands of uneven small systems in one plan, FP64
        {"name": "batch64_4096", "kind": "batch", "count": 4096, "nmin": 16, "nmax": 512, "mode": 0},
        # the same with FP32 factors and FP64 refinement
        {"name": "batch32_4096", "kind": "batch", "count": 4096, "nmin": 16, "nmax": 512, "mode": 1},
        # mixed-precision solve with refinement
        {"name": "ir_n8192_r4", "kind": "ir", "n": 8192, "nrhs": 4, "fmt": "bf16x3"},
        # explicit inverse from the factors
        {"name": "getri_n3000", "kind": "getri", "n": 3000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gesv", "gesv", "gesv", "getrf", "getrs", "getrs", "pdgesv", "batch", "ir", "getri"])
    if kind == "gesv":
        return {"kind": kind, "n": _log(rng, 8, 16000), "nrhs": rng.randint(1, 16),
                "nb": rng.choice([0, 64, 128, 256])}
    if kind == "getrf":
        return {"kind": kind, "m": _log(rng, 32, 9000), "n": _log(rng, 32, 9000), "nb": rng.choice([0, 64, 256])}
    if kind == "getrs":
        return {"kind": kind, "n": _log(rng, 64, 12000), "nrhs": _log(rng, 1, 64), "trans": rng.choice(["N", "T"])}
    if kind == "pdgesv":
        return {"kind": kind, "n": _log(rng, 64, 4000), "nrhs": rng.randint(1, 8), "nb": rng.choice([32, 64, 256])}
    if kind == "batch":
        lo = rng.randint(1, 64)
        return {"kind": kind, "count": _log(rng, 100, 4000), "nmin": lo, "nmax": rng.randint(lo + 8, 512),
                "mode": rng.randint(0, 1)}
    if kind == "ir":
        return {"kind": kind, "n": _log(rng, 700, 10000), "nrhs": rng.randint(1, 4),
                "fmt": rng.choice(["bf16x3", "fp16"])}
    return {"kind": kind, "n": _log(rng, 64, 4000)}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _matrix(m, n, g):
    """m x n column-major (an n x m tensor): noise plus a shift on a permuted diagonal."""
    a = torch.rand((n, m), dtype=F64, device="cuda", generator=g).sub_(0.5)
    k = min(m, n)
    rows = torch.randperm(m, device="cuda", generator=g)[:k]
    a[torch.arange(k, device="cuda"), rows] += 0.5 * math.sqrt(m)
    return a


def _rhs(n, nrhs, g):
    return torch.rand((nrhs, n), dtype=F64, device="cuda", generator=g).sub_(0.5)


def _batch_inputs(case, seed):
    """Orders, right-hand-side counts and the packed matrices and right-hand sides of a batch."""
    r = np.random.default_rng(case["count"])  # the shapes belong to the case, the values to the seed
    ns = r.integers(case["nmin"], case["nmax"] + 1, size=case["count"])
    rs = r.integers(1, 9, size=case["count"])
    r = np.random.default_rng(seed)
    ao = np.concatenate([[0], np.cumsum(ns * ns)])
    bo = np.concatenate([[0], np.cumsum(ns * rs)])
    g = _gen(seed)
    a = torch.rand(int(ao[-1]), dtype=F64, device="cuda", generator=g).sub_(0.5)
    b = torch.rand(int(bo[-1]), dtype=F64, device="cuda", generator=g).sub_(0.5)
    at = np.concatenate([o + np.arange(n) * n + r.permutation(n) for o, n in zip(ao, ns)])
    shift = np.repeat(0.5 * np.sqrt(ns), ns)
    a[torch.from_numpy(at).cuda()] += torch.from_numpy(shift).cuda()
    return ns, rs, ao, bo, a, b


def _desc(ctxt, m, n, nb):
    return np.array([1, ctxt, m, n, nb, nb, 0, 0, max(1, m)], dtype=np.int32)


class _Plan(sl.BatchPlan):
    """A plan that gives its device memory back with its last reference."""

    def __del__(self):
        self.close()


_ctxt = None


def _context():
    global _ctxt
    if _ctxt is None:
        _ctxt = sl.blacs_gridinit(1, 1)
    return _ctxt


def _inputs(case, seed):
    """The matrix and right-hand sides of a single-system case."""
    g = _gen(seed)
    n = case["n"]
    a = _matrix(case.get("m", n), n, g)
    return a, _rhs(n, case["nrhs"], g) if "nrhs" in case else None


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        ns, rs, ao, bo, a, b = _batch_inputs(case, seed)
        x = torch.zeros_like(b)
        s.update(A=a, B=b, X=x)
        systems = [(a.data_ptr() + 8 * int(ao[i]), int(n), int(n), b.data_ptr() + 8 * int(bo[i]), int(n), int(rs[i]),
                    x.data_ptr() + 8 * int(bo[i]), int(n)) for i, n in enumerate(ns)]
        s["plan"] = _Plan(systems, mode=case["mode"])
        return s
    a, b = _inputs(case, seed)
    n = case["n"]
    if kind == "pdgesv":
        s["A0"], s["B0"] = (np.asfortranarray(t.cpu().numpy().T) for t in (a, b))
        s["A"], s["B"] = s["A0"].copy(order="F"), s["B0"].copy(order="F")
        s["ipiv"] = np.zeros(n + case["nb"], dtype=np.int32)
        s["da"] = _desc(_context(), n, n, case["nb"])
        s["db"] = _desc(_context(), n, case["nrhs"], case["nb"])
        return s
    s["ipiv"] = torch.zeros(min(case.get("m", n), n), dtype=torch.int32, device="cuda")
    if kind in ("getrs", "getri"):
        torch.cuda.synchronize()
        if sl.dgetrf_dev(n, n, a.data_ptr(), n, s["ipiv"].data_ptr()) != 0:
            raise RuntimeError("factorization failed")
    s["A0"], s["B0"] = a, b
    if kind in ("gesv", "getrf", "getri"):
        s["A"] = torch.empty_like(a)
    if kind in ("gesv", "getrs"):
        s["B"] = torch.empty_like(b)
    if kind == "ir":
        s["X"] = torch.zeros_like(b)
    return s


def _ok(info):
    if info != 0:
        raise RuntimeError(f"INFO={info}")


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "batch":
        s["plan"].execute()
        return s["X"]
    n = c["n"]
    if kind == "pdgesv":
        np.copyto(s["A"], s["A0"])
        np.copyto(s["B"], s["B0"])
        _ok(sl.pdgesv(n, c["nrhs"], s["A"], 1, 1, s["da"], s["ipiv"], s["B"], 1, 1, s["db"]))
        return {"A": s["A"], "ipiv": s["ipiv"][:n], "X": s["B"]}
    stream = torch.cuda.current_stream().cuda_stream
    ip = s["ipiv"].data_ptr()
    if kind == "ir":
        info, _, _ = sl.dgesv_ir_dev(n, c["nrhs"], s["A0"].data_ptr(), n, ip, s["B0"].data_ptr(), n,
                                     s["X"].data_ptr(), n, fmt=c["fmt"], stream=stream)
        _ok(info)
        return {"X": s["X"]}
    if kind == "getrs":
        s["B"].copy_(s["B0"])
        _ok(sl.dgetrs_dev(c["trans"], n, c["nrhs"], s["A0"].data_ptr(), n, ip, s["B"].data_ptr(), n, stream=stream))
        return {"X": s["B"]}
    s["A"].copy_(s["A0"])
    if kind == "getri":
        _ok(sl.lib().sl1x1_dgetri_dev(n, s["A"].data_ptr(), n, ip, stream))
        return {"inv": s["A"]}
    if kind == "getrf":
        m = c["m"]
        _ok(sl.dgetrf_dev(m, n, s["A"].data_ptr(), m, ip, c["nb"], stream=stream))
        return {"A": s["A"], "ipiv": s["ipiv"]}
    s["B"].copy_(s["B0"])
    _ok(sl.dgesv_dev(n, c["nrhs"], s["A"].data_ptr(), n, ip, s["B"].data_ptr(), n, c["nb"], stream=stream))
    return {"A": s["A"], "ipiv": s["ipiv"], "X": s["B"]}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # expected values over the uniform distribution of the orders
        n = np.arange(case["nmin"], case["nmax"] + 1, dtype=np.float64)
        return {"bytes": float(case["count"] * np.mean(8 * (n * n + 2 * 4.5 * n))),
                "flops": float(case["count"] * np.mean(2 * n**3 / 3 + 2 * 4.5 * n * n))}
    n = case["n"]
    r = case.get("nrhs", 0)
    lu = 2 * n**3 / 3
    if kind == "getrf":
        m = case["m"]
        k = min(m, n)
        return {"bytes": 16 * m * n + 4 * k, "flops": 2 * m * n * k - (m + n) * k * k + 2 * k**3 / 3}
    if kind == "getrs":
        return {"bytes": 8 * n * n + 16 * n * r, "flops": 2 * n * n * r}
    if kind == "getri":
        return {"bytes": 16 * n * n, "flops": 4 * n**3 / 3}
    if kind == "ir":
        return {"bytes": 8 * n * n + 16 * n * r, "flops": lu + 2 * n * n * r}
    return {"bytes": 16 * n * n + 16 * n * r + 4 * n, "flops": lu + 2 * n * n * r}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ns, rs, ao, bo, a, b = _batch_inputs(case, seed)
        a, b = a.cpu().numpy(), b.cpu().numpy()
        x = np.empty_like(b)
        for i, (n, r) in enumerate(zip(ns, rs)):
            m = a[ao[i]:ao[i + 1]].reshape(n, n).T
            x[bo[i]:bo[i + 1]] = np.linalg.solve(m, b[bo[i]:bo[i + 1]].reshape(r, n).T).T.reshape(-1)
        return x
    a, b = _inputs(case, seed)
    if kind == "getri":
        return {"inv": torch.linalg.inv(a)}
    if kind in ("ir", "getrs"):
        m = a if case.get("trans") == "T" else a.T
        return {"X": torch.linalg.solve(m, b.T).T.contiguous()}
    lu, piv = torch.linalg.lu_factor(a.T)
    out = {"A": lu.T.contiguous(), "ipiv": piv}
    if kind == "getrf":
        return out
    out["X"] = torch.linalg.lu_solve(lu, piv, b.T).T.contiguous()
    if kind == "pdgesv":
        return {"A": np.asfortranarray(out["A"].cpu().numpy().T), "ipiv": piv.cpu().numpy(),
                "X": np.asfortranarray(out["X"].cpu().numpy().T)}
    return out
