"""Workloads for timing the library through its public entry points.

Each case is one call as a program that uses lu2_b200 makes it, on inputs made
from a seed: the plain FP64 solve on the device over its range of orders, the
drop-in `lumcolumn` on host memory, the re-solve from stored factors, the two
precision forms, the two arithmetics of the batching form, and the device
DGEMM.  `listed()` names the fixed ones, `draw(rng)` gives more of the same
ranges, `prepare` / `run` / `work` / `exact` make, run, count and check one.

All matrices are uniform in [-0.5, 0.5), lu2's own distribution, with two
variations that the precision and batching forms need to have solutions that
are determined to many digits: `dominant` puts each row's absolute sum on the
diagonal (the precision forms' workload), and the batch adds 0.5 sqrt(n) to one
entry per row, off the diagonal so that rows have to be exchanged.
"""
import math

import numpy as np
import torch

import lu2_b200 as L

# the batching form's largest order here, and its share of systems with several right-hand sides
BATCH_NMIN, BATCH_MULTI, BATCH_NRHS = 16, 0.1, 8

_context = None


def _ctx():
    """The one context a program keeps for its device, on torch's stream."""
    global _context
    if _context is None:
        _context = L.Context(0)
        _context.set_stream(torch.cuda.current_stream().cuda_stream)
    return _context


def listed():
    return [
        # a small dense system on the device: latency and launches
        {"name": "lu_n384", "kind": "lu", "n": 384, "nb": 64, "nrhs": 1},
        # a small system of an odd order with several right-hand sides
        {"name": "lu_n1001_r7", "kind": "lu", "n": 1001, "nb": 64, "nrhs": 7},
        # lu2's own program: lumcolumn on malloc'd host memory, N=2048, block 64
        {"name": "lumcolumn_n2048", "kind": "lumcolumn", "n": 2048, "nb": 64},
        # an ordinary order that is no multiple of anything
        {"name": "lu_n3333_r3", "kind": "lu", "n": 3333, "nb": 128, "nrhs": 3},
        # the order at which the device is compared with the host's lu2
        {"name": "lu_n8192", "kind": "lu", "n": 8192, "nb": 256, "nrhs": 1},
        # a large system (4.8 GB)
        {"name": "lu_n24576", "kind": "lu", "n": 24576, "nb": 256, "nrhs": 1},
        # new right-hand sides for a matrix that was factored before
        {"name": "resolve_n6144_r4", "kind": "resolve", "n": 6144, "nb": 256, "nrhs": 4},
        # BF16 factorization with FP64 refinement
        {"name": "mixed_n12288", "kind": "mixed", "n": 12288, "nb": 256},
        # E4M3 factorization with GMRES refinement
        {"name": "gmres_fp8_n10240", "kind": "gmres", "n": 10240, "nb": 256},
        # thousands of uneven systems, FP64
        {"name": "batch_fp64_4000", "kind": "batch", "count": 4000, "nmax": 512, "ir": False},
        # the same with FP32 factors and FP64 refinement
        {"name": "batch_ir_2000", "kind": "batch", "count": 2000, "nmax": 512, "ir": True},
        # C -= A B, the offloaded product, K of a wide panel
        {"name": "dgemm_5000x4000x512", "kind": "dgemm", "m": 5000, "n": 4000, "k": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lu", "lu", "lu", "lumcolumn", "resolve", "mixed", "gmres", "batch", "batch", "dgemm"])
    if kind == "lu":
        n = _log(rng, 256, 16384)
        return {"kind": kind, "n": n, "nb": 64 if n < 2048 else rng.choice([64, 128, 256]), "nrhs": rng.randint(1, 8)}
    if kind == "lumcolumn":
        return {"kind": kind, "n": _log(rng, 512, 3072), "nb": rng.choice([64, 128])}
    if kind == "resolve":
        return {"kind": kind, "n": _log(rng, 1024, 10240), "nb": rng.choice([64, 128, 256]), "nrhs": rng.randint(1, 8)}
    if kind in ("mixed", "gmres"):
        return {"kind": kind, "n": _log(rng, 2048, 14336), "nb": rng.choice([128, 256])}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 300, 4000), "nmax": rng.choice([64, 128, 256, 400, 512]),
                "ir": rng.random() < 0.4}
    return {"kind": kind, "m": _log(rng, 256, 8192), "n": _log(rng, 256, 8192), "k": rng.choice([64, 100, 256, 512, 1024])}


# ---------------------------------------------------------------------------
# inputs, the same for `prepare` and `exact`


def _uniform(shape, gen):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen) - 0.5


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _system(case, seed, nrhs, dominant=False):
    """A (n x n) and B (n x nrhs)."""
    gen = _gen(seed)
    n = case["n"]
    a = _uniform((n, n), gen)
    if dominant:
        a.diagonal().copy_(a.abs().sum(1))
    return a, _uniform((n, nrhs), gen)


def _batch_shape(case):
    """Orders, right-hand sides and storage (offset, row stride) of every system."""
    rng = np.random.default_rng([case["count"], case["nmax"]])
    lo, hi = math.log(BATCH_NMIN), math.log(case["nmax"] + 1)
    n = np.clip(np.exp(rng.uniform(lo, hi, case["count"])).astype(np.int64), BATCH_NMIN, case["nmax"])
    r = np.where(rng.random(case["count"]) < BATCH_MULTI, BATCH_NRHS, 1)
    ld = (n + r + 1) & ~1
    off = np.concatenate([[0], np.cumsum(n * ld)])
    return n, r, ld, off


def _batch_data(case, seed):
    """The packed systems: row-major, right-hand sides in the columns after n."""
    n, r, ld, off = _batch_shape(case)
    data = _uniform((int(off[-1]),), _gen(seed))
    row = np.arange(int(n.sum())) - np.repeat(np.cumsum(n) - n, n)
    order = np.repeat(n, n)
    at = np.repeat(off[:-1], n) + row * np.repeat(ld, n) + (row + order // 3) % order
    data[torch.from_numpy(at).cuda()] += torch.from_numpy(0.5 * np.sqrt(order)).cuda()
    return data, n, r, ld, off


class _DeviceArray:
    """A view of device memory the library owns."""

    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 2}


# ---------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    ctx = _ctx()
    if kind == "lu":
        n, nrhs = case["n"], case["nrhs"]
        a, b = _system(case, seed, nrhs)
        ld = L.device_ld(n, nrhs)
        given = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
        given[:, :n] = a
        given[:, n:n + nrhs] = b
        return {"case": case, "ctx": ctx, "ld": ld, "given": given, "a": torch.empty_like(given),
                "ipiv": torch.zeros(n, dtype=torch.int32, device="cuda")}
    if kind == "lumcolumn":
        n = case["n"]
        a, b = _system(case, seed, 1)
        given = np.zeros((n, L.rdim(n)))
        given[:, :n] = a.cpu().numpy()
        given[:, n] = b[:, 0].cpu().numpy()
        return {"case": case, "given": given, "a": np.empty_like(given), "x": np.zeros(n),
                "pv": np.zeros(case["nb"], dtype=np.int32)}
    if kind == "resolve":
        n, nrhs = case["n"], case["nrhs"]
        a, b = _system(case, seed, nrhs)
        ld = L.device_ld(n, 0)
        f = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
        f[:, :n] = a
        ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ctx.factor(f, n, ld, case["nb"], 0, L.PIVOT_PARTIAL, ipiv)
        return {"case": case, "ctx": ctx, "ld": ld, "f": f, "ipiv": ipiv, "b": b, "x": torch.empty_like(b)}
    if kind in ("mixed", "gmres"):
        n = case["n"]
        a, b = _system(case, seed, 1, dominant=True)
        ld = L.device_ld(n, 0)
        full = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
        full[:, :n] = a
        return {"case": case, "ctx": ctx, "ld": ld, "a": full, "b": b[:, 0].contiguous(),
                "x": torch.zeros(n, dtype=torch.float64, device="cuda")}
    if kind == "batch":
        data, n, r, ld, off = _batch_data(case, seed)
        batch = L.Batch(ctx, n.astype(np.int32), r.astype(np.int32))
        base, _ = batch.system(0)
        if any(batch.system(i) != (base + 8 * int(off[i]), int(ld[i])) for i in (1, len(n) // 2, len(n) - 1)):
            raise RuntimeError("the batch's storage is not packed as expected")
        view = torch.as_tensor(_DeviceArray(base, int(off[-1])), device="cuda")
        view.copy_(data)
        torch.cuda.synchronize()
        if case["ir"]:
            batch.set_mode(L.BATCH_FP32_IR)
        batch.autotune()  # keeps a copy of the systems, too
        # where the solutions are: rows in order, each with its right-hand sides
        rows = int((n * r).sum())
        sys_of = np.repeat(np.arange(len(n)), n * r)
        k = np.arange(rows) - np.repeat(np.cumsum(n * r) - n * r, n * r)
        at = off[sys_of] + (k // r[sys_of]) * ld[sys_of] + n[sys_of] + k % r[sys_of]
        return {"case": case, "batch": batch, "view": view, "at": torch.from_numpy(at).cuda()}
    m, n, k = case["m"], case["n"], case["k"]
    gen = _gen(seed)
    a, b, c = _uniform((m, k), gen), _uniform((k, n), gen), _uniform((m, n), gen)
    return {"case": case, "ctx": ctx, "a": a, "b": b, "given": c, "c": torch.empty_like(c)}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "lumcolumn":
        np.copyto(s["a"], s["given"])
        L.lumcolumn(s["a"], s["x"], case["nb"], s["pv"])
        return {"x": s["x"], "factors": s["a"][:, :case["n"]], "pv": s["pv"]}
    if kind == "batch":
        s["batch"].restore()
        info = s["batch"].solve()
        return {"x": s["view"][s["at"]], "info": info}
    ctx = s["ctx"]
    if kind == "lu":
        n, nrhs = case["n"], case["nrhs"]
        s["a"].copy_(s["given"])
        status = ctx.lusolve(s["a"], n, s["ld"], case["nb"], nrhs, L.PIVOT_PARTIAL, s["ipiv"])
        return {"x": s["a"][:, n:n + nrhs], "factors": s["a"][:, :n], "ipiv": s["ipiv"], "status": status}
    if kind == "resolve":
        s["x"].copy_(s["b"])
        ctx.solve(s["f"], case["n"], s["ld"], case["nb"], s["ipiv"], s["x"], case["nrhs"], case["nrhs"])
        return {"x": s["x"]}
    if kind == "mixed":
        got = ctx.mixed_solve(s["a"], case["n"], s["ld"], s["b"], s["x"], case["nb"])
        return {"x": s["x"], "status": got["status"], "iterations": got["iterations"]}
    if kind == "gmres":
        got = ctx.gmres_solve(s["a"], case["n"], s["ld"], s["b"], s["x"], case["nb"])
        return {"x": s["x"], "status": got["status"], "refinements": got["refinements"],
                "gmres_iterations": got["gmres_iterations"]}
    s["c"].copy_(s["given"])
    ctx.dgemm(case["m"], case["n"], case["k"], -1.0, s["a"], case["k"], s["b"], case["n"], 1.0, s["c"], case["n"])
    return {"c": s["c"]}


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    2/3 n^3 + 2 n^2 per right-hand side for a factorization and solve, 2 n^2 per
    right-hand side for a solve alone, 2 m n k for a product."""
    kind = case["kind"]
    if kind == "batch":
        n, r, _, _ = _batch_shape(case)
        n, r = n.astype(float), r.astype(float)
        return {"bytes": float((8 * n * n + 16 * n * r).sum()),
                "flops": float((2 / 3 * n**3 + 2 * n * n * r).sum())}
    if kind == "dgemm":
        m, n, k = float(case["m"]), float(case["n"]), float(case["k"])
        return {"bytes": 8 * (m * k + k * n + 2 * m * n), "flops": 2 * m * n * k}
    n, r = float(case["n"]), float(case.get("nrhs", 1))
    if kind == "resolve":
        return {"bytes": 8 * n * n + 16 * n * r, "flops": 2 * n * n * r}
    if kind in ("mixed", "gmres"):
        return {"bytes": 8 * n * n + 16 * n, "flops": 2 / 3 * n**3 + 2 * n * n}
    return {"bytes": 16 * n * (n + r), "flops": 2 / 3 * n**3 + 2 * n * n * r}


def exact(case, seed):
    """The solutions (and the product) in 64 bits; the factors and pivots have
    lu2's own layout and no counterpart in plain torch."""
    kind = case["kind"]
    if kind == "dgemm":
        m, n, k = case["m"], case["n"], case["k"]
        gen = _gen(seed)
        a, b, c = _uniform((m, k), gen), _uniform((k, n), gen), _uniform((m, n), gen)
        return {"c": c - a @ b}
    if kind == "batch":
        data, n, r, ld, off = _batch_data(case, seed)
        x = torch.empty(int((n * r).sum()), dtype=torch.float64, device="cuda")
        first = np.cumsum(n * r) - n * r
        pad = (n + 31) // 32 * 32  # solved in groups of one padded order (identity beyond n)
        for p in np.unique(pad):
            for part in np.array_split(np.flatnonzero(pad == p), max(1, int((pad == p).sum()) // 512)):
                a = torch.eye(int(p), dtype=torch.float64, device="cuda").repeat(len(part), 1, 1)
                b = torch.zeros((len(part), int(p), BATCH_NRHS), dtype=torch.float64, device="cuda")
                for q, i in enumerate(part):
                    ni, ri = int(n[i]), int(r[i])
                    full = data[int(off[i]):int(off[i]) + ni * int(ld[i])].view(ni, int(ld[i]))
                    a[q, :ni, :ni] = full[:, :ni]
                    b[q, :ni, :ri] = full[:, ni:ni + ri]
                sol = torch.linalg.solve(a, b)
                for q, i in enumerate(part):
                    ni, ri = int(n[i]), int(r[i])
                    x[int(first[i]):int(first[i]) + ni * ri] = sol[q, :ni, :ri].reshape(-1)
        return {"x": x, "info": None}
    dominant = kind in ("mixed", "gmres")
    a, b = _system(case, seed, case.get("nrhs", 1), dominant)
    x = torch.linalg.solve(a, b)
    if kind == "lu":
        return {"x": x, "factors": None, "ipiv": None, "status": None}
    if kind == "lumcolumn":
        return {"x": x[:, 0], "factors": None, "pv": None}
    if kind == "resolve":
        return {"x": x}
    return {"x": x[:, 0]}
