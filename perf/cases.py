"""Performance cases of the matrix-profile framework.

Each case is one call that a user's program makes through the public entry
points of ``thesiscode_b200``: whole self-joins in the three numeric forms, the
approximate PreSCRIMP profile, the block kernel that the reference's drivers
call, a batch of many series and a burst of requests to the server.  Series are
seeded random walks (the generators of ``thesiscode_b200.workloads``), the data
every workload of this path is defined on.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import thesiscode_b200 as mp
from thesiscode_b200 import workloads

WINDOWS = (32, 64, 128, 256, 512, 1024)


def listed():
    return [
        # The smallest calls: one short series, arrays in host memory, where the
        # number of launches and the serial parts of the preparation count.
        {"name": "fp64_small", "kind": "join", "form": "fp64", "n": 2500, "m": 100, "k": 0,
         "host": True},
        {"name": "fp32_small", "kind": "join", "form": "fp32", "n": 4099, "m": 64, "k": 0,
         "host": True},
        # An ordinary series: the reference's own CPU case (65,536 samples, m = 400).
        {"name": "fp64_c1", "kind": "join", "form": "fp64", "n": 65536, "m": 400, "k": 0,
         "host": False},
        {"name": "fp32_c1", "kind": "join", "form": "fp32", "n": 65536, "m": 400, "k": 0,
         "host": False},
        # The long single series of the headline (1,048,576 samples, m = 256).
        {"name": "fp64_c2", "kind": "join", "form": "fp64", "n": 1048576, "m": 256, "k": 0,
         "host": False},
        {"name": "fp32_c2", "kind": "join", "form": "fp32", "n": 1048576, "m": 256, "k": 1024,
         "host": False},
        # A caller that wants a smaller error: long windows, short re-anchor interval.
        {"name": "fp32_k256", "kind": "join", "form": "fp32", "n": 300007, "m": 1000, "k": 256,
         "host": False},
        # Data with planted motifs and constant stretches, in the guarded form.
        {"name": "guarded_stress", "kind": "join", "form": "guarded", "n": 262144, "m": 1024,
         "k": 0, "host": False},
        # SCRIMP++'s anytime first look at a long series.
        {"name": "prescrimp", "kind": "prescrimp", "n": 200003, "m": 256, "stride": 0.25},
        # The reference's kernel interface as its driver calls it: one block of
        # --blocklen diagonals, host arrays, profile views that alias.
        {"name": "block_kernel", "kind": "block", "n": 65536, "m": 400, "blocklen": 500,
         "diag": 20101},
        # A collection of FP32 series of uneven length solved as one plan.
        {"name": "batch", "kind": "batch", "count": 24, "lo": 2048, "hi": 262144, "shape_seed": 3},
        # A burst of requests to the server, short and long ones mixed.
        {"name": "serve_burst", "kind": "serve", "count": 16, "lo": 1024, "hi": 131072,
         "shape_seed": 4},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["join", "join", "join", "join", "prescrimp", "block", "batch", "serve"])
    if kind == "join":
        form = rng.choice(["fp64", "fp32", "fp32", "guarded"])
        n = _log_int(rng, 1500, 900000)
        m = rng.choice([w for w in WINDOWS if 8 * w <= n] + [rng.randint(20, min(1100, n // 8))])
        k = 0
        if form != "fp64":
            k = rng.choice([0, 1024, 512, 256, 64])
            # an anchor costs m FP64 operations per k columns: the short
            # intervals are for series that are not too long
            n = min(n, int(900000 * math.sqrt(min(1.0, 2.0 * max(k, 512) / (m + 512)))))
            n = min(n, 150000) if k == 64 else n
            n = min(n, 400000) if form == "guarded" else n
        if form == "guarded":
            n = max(n, 128 * m)  # room for the planted stretches
        return {"kind": "join", "form": form, "n": n, "m": m, "k": k,
                "host": rng.random() < 0.3}
    if kind == "prescrimp":
        n = _log_int(rng, 4000, 300000)
        m = rng.choice([w for w in WINDOWS if 8 * w <= n] + [rng.randint(40, min(900, n // 8))])
        return {"kind": "prescrimp", "n": n, "m": m, "stride": rng.choice([0.25, 0.25, 0.5, 1.0, 2.0])}
    if kind == "block":
        n = _log_int(rng, 4000, 300000)
        m = rng.choice([w for w in WINDOWS if 8 * w <= n])
        return {"kind": "block", "n": n, "m": m, "blocklen": rng.choice([100, 500, 500, 777, 1000]),
                "diag": rng.randint(m // 4 + 1, n // 2)}
    count = rng.randint(4, 30)
    hi = _log_int(rng, 20000, 200000)
    return {"kind": kind, "count": count, "lo": 1024 if kind == "serve" else 2048, "hi": hi,
            "shape_seed": rng.randint(0, 1 << 20)}


def _shapes(case):
    """(n, m) of each series of a batch or burst; fixed by the case, not by the seed."""
    rng = np.random.default_rng(case["shape_seed"])
    lens = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["count"])).astype(int)
    ms = rng.choice([64, 128, 256] if case["kind"] == "batch" else WINDOWS, size=case["count"])
    return [(max(int(n), 2 * int(m)), int(m)) for n, m in zip(lens, ms)]


def _form(case):
    return {"fp64": mp.FP64, "fp32": mp.FP32_REANCHOR, "guarded": mp.FP32_GUARDED}[case["form"]]


def _series(case, seed):
    if case["kind"] == "join" and case["form"] == "guarded":
        return workloads.c3(case["n"], case["m"], seed=seed)[0]
    return workloads.random_walk(case["n"], seed)


def _walks(case, seed):
    dtype = np.float32 if case["kind"] == "batch" else np.float64
    return [workloads.random_walk(n, seed * 1009 + i).astype(dtype)
            for i, (n, _) in enumerate(_shapes(case))]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("join", "prescrimp"):
        x = _series(case, seed)
        pl = case["n"] - case["m"] + 1
        s["ctx"] = mp.Context(0)
        if case.get("host"):
            s["x"], s["out"] = x, (np.empty(pl), np.empty(pl, dtype=np.int64))
        else:
            s["x"] = torch.from_numpy(x).cuda()
            s["out"] = (torch.empty(pl, dtype=torch.float64, device="cuda"),
                        torch.empty(pl, dtype=torch.int64, device="cuda"))
        # the context's scratch is part of the handle that a program keeps
        _call(s)
    elif kind == "block":
        x, m, g = _series(case, seed), case["m"], case["diag"]
        s["ctx"] = mp.Context(0)
        s["mu"], s["sinv"] = s["ctx"].window_stats(x, m)
        s["q"] = s["ctx"].first_qt(x, m, g, min(g + case["blocklen"], x.size - m + 1))
        s["x"] = np.append(x, 0.0)  # the update after a diagonal's last cell reads A[n]
        s["pl"] = x.size - m + 1
        _call(s)
    elif kind == "batch":
        s["ctx"] = mp.Context(0)
        s["series"] = _walks(case, seed)
        shapes = _shapes(case)
        s["batch"] = mp.Batch(s["ctx"], [n for n, _ in shapes], [m for _, m in shapes])
        s["out"] = s["batch"].outputs()
        _call(s)
    else:
        s["series"] = _walks(case, seed)
        s["server"] = mp.Server(0, mem_budget_bytes=8 << 30, slots=32)
        _call(s)
    return s


def _call(s):
    case = s["case"]
    kind, m = case["kind"], case.get("m")
    if kind == "join":
        return s["ctx"].selfjoin(s["x"], m, precision=_form(case), reanchor_k=case["k"],
                                 out=s["out"])
    if kind == "prescrimp":
        return s["ctx"].prescrimp(s["x"], m, case["stride"], out=s["out"])
    if kind == "block":
        g, pl = case["diag"], s["pl"]
        t, nd = pl - g, s["q"].size
        prof, idx, q = np.full(pl, -1.0), np.zeros(pl, dtype=np.int64), s["q"].copy()
        s["ctx"].eval_diag_block_triangle(
            prof[:t], idx[:t], prof[g:], idx[g:], q, nd, t, s["x"], s["x"][g:], m, s["sinv"],
            s["mu"], s["sinv"][g:], s["mu"][g:], g, 0)
        return prof, idx, q
    if kind == "batch":
        return s["batch"].run(s["series"], out=s["out"])
    tickets = [s["server"].submit(x, m) for x, (_, m) in zip(s["series"], _shapes(case))]
    return [s["server"].collect(t)[1] for t, _ in tickets]


def run(state):
    r = _call(state)
    if state["case"]["kind"] == "block":
        return list(r)
    if isinstance(r, list):
        return [[p.dist2, p.index] for p in r]
    return [r.dist2, r.index]


def _cells(n, m):
    d = max(n - m + 1 - m // 4 - 1, 0)
    return d * (d + 1) // 2


def work(case):
    kind = case["kind"]
    # a cell: two fused operations for the running dot product, one fused
    # operation and two products for its score
    if kind == "join":
        n, m = case["n"], case["m"]
        return {"bytes": 8 * n + 16 * (n - m + 1), "flops": 8 * _cells(n, m)}
    if kind == "prescrimp":
        n, m = case["n"], case["m"]
        pl, step = n - m + 1, int(math.floor(case["stride"] * m))
        q = (pl + step - 1) // step
        # dot products between blocks of min(step, m) samples, shared by the
        # queries that contain them
        return {"bytes": 8 * n + 16 * pl, "flops": 2 * q * pl * min(step, m)}
    if kind == "block":
        n, m, g = case["n"], case["m"], case["diag"]
        t = n - m + 1 - g
        nd = min(case["blocklen"], t)
        return {"bytes": 8 * (2 * n + 6 * t) + 32 * t,
                "flops": 8 * (nd * t - nd * (nd - 1) // 2)}
    esz = 4 if kind == "batch" else 8
    shapes = _shapes(case)
    return {"bytes": sum(esz * n + 16 * (n - m + 1) for n, m in shapes),
            "flops": sum(8 * _cells(n, m) for n, m in shapes)}


# ---- what the calls return, in plain 64-bit torch ---------------------------

def _windows(x, m):
    """Unit-norm centred windows [PL, m] on the GPU; rows of constant windows are 0."""
    w = torch.from_numpy(np.asarray(x, dtype=np.float64)).cuda().unfold(0, m, 1)
    flat = w.amax(1) == w.amin(1)
    z = w - w.mean(1, keepdim=True)
    z /= torch.where(flat, torch.ones_like(z[:, 0]), z.norm(dim=1)).unsqueeze(1)
    z[flat] = 0.0
    return z, flat


def _join_dist2(x, m):
    """Squared distance of every window to its nearest neighbour outside m/4."""
    z, flat = _windows(x, m)
    pl, excl = z.shape[0], m // 4
    best = torch.full((pl,), -math.inf, dtype=torch.float64, device="cuda")
    z_flat = flat.any()
    step = 4096
    for a in range(0, pl, step):
        b = min(a + step, pl)
        c0 = a + excl + 1
        if c0 >= pl:
            break
        c = z[a:b] @ z[c0:].T
        near = torch.arange(c0, min(c0 + step, pl), device="cuda") - \
            torch.arange(a, b, device="cuda").unsqueeze(1) <= excl
        c[:, :near.shape[1]].masked_fill_(near, -math.inf)
        if z_flat:
            c[flat[a:b]] = -math.inf
            c[:, flat[c0:]] = -math.inf
        best[a:b] = torch.maximum(best[a:b], c.amax(1))
        best[c0:] = torch.maximum(best[c0:], c.amax(0))
    none = m * best <= -1.0
    return torch.where(none, torch.full_like(best, 2.0 * m + 2.0), 2.0 * m * (1.0 - best)).cpu()


def _prescrimp_dist2(x, m, stride):
    z, flat = _windows(x, m)
    pl, excl, step = z.shape[0], m // 4, int(math.floor(stride * m))
    prof = torch.full((pl,), math.inf, dtype=torch.float64, device="cuda")
    queries = torch.arange(0, pl, step, device="cuda")
    js = torch.arange(pl, device="cuda")
    for q0 in range(0, queries.numel(), 2048):
        i = queries[q0:q0 + 2048]
        d = 2.0 * m * (1.0 - z[i] @ z.T)
        d.masked_fill_((js - i.unsqueeze(1)).abs() < excl, math.inf)
        prof = torch.minimum(prof, d.amin(0))
        best, j = d.min(1)
        prof[i] = torch.minimum(prof[i], best)
        for k in range(-step + 1, step):  # the walk along each query's best diagonal
            p, r = i + k, j + k
            ok = (p >= 0) & (r >= 0) & (p < pl) & (r < pl) & torch.isfinite(best)
            p, r = p[ok], r[ok]
            v = 2.0 * m * (1.0 - (z[p] * z[r]).sum(1))
            prof.scatter_reduce_(0, p, v, "amin")
            prof.scatter_reduce_(0, r, v, "amin")
    return prof.cpu()


def _block_scores(x, m, g, nd):
    """Best score m * correlation per window over diagonals [g, g + nd), from -1."""
    z, _ = _windows(x, m)
    pl = z.shape[0]
    prof = torch.full((pl,), -1.0, dtype=torch.float64, device="cuda")
    for d in range(g, min(g + nd, pl)):
        s = m * (z[:pl - d] * z[d:]).sum(1)
        prof[:pl - d] = torch.maximum(prof[:pl - d], s)
        prof[d:] = torch.maximum(prof[d:], s)
    return prof.cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "join":
        if float(case["n"]) ** 2 * case["m"] > 1.5e14:
            return None  # over about 20 seconds
        return [_join_dist2(_series(case, seed), case["m"]), None]
    if kind == "prescrimp":
        if float(case["n"]) ** 2 / case["stride"] > 5e13:
            return None
        return [_prescrimp_dist2(_series(case, seed), case["m"], case["stride"]), None]
    if kind == "block":
        t = case["n"] - case["m"] + 1 - case["diag"]
        if float(t) * case["m"] * case["blocklen"] > 2e12:
            return None
        nd = min(case["blocklen"], t)
        return [_block_scores(_series(case, seed), case["m"], case["diag"], nd), None, None]
    shapes = _shapes(case)
    if sum(float(n) ** 2 * m for n, m in shapes) > 1.5e14:
        return None
    return [[_join_dist2(x, m), None] for x, (_, m) in zip(_walks(case, seed), shapes)]
