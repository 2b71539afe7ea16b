"""Workloads of the graph codes, each one pass through the public entry points.

A case names the codes it calls, the graph family and its size, and where the
graph lives; everything else follows from the seed.  Graphs are made on the
GPU with torch (R-MAT with the quadrant probabilities of ecl_gen_rmat, the
4-neighbour grid with deleted edges of ecl_gen_grid, and G(n, m) graphs with
the average degree of ecl_gen_er), because making an R-MAT-22 graph on the host
takes longer than solving it thousands of times.

Kinds of case (the "kind" of a case):
  solve  - the single-graph solvers on one graph, device- or host-resident
  apsp   - all-pairs shortest paths of one weighted directed graph
  batch  - the batched engine: many small graphs, one run, every result read
  serve  - the request server: a Poisson stream over resident graphs
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "ecl-suite_b200"))

import ecl_b200 as ecl  # noqa: E402

WEIGHT_MAX = 1 << 20
CODES = ("cc", "mis", "gc", "mst", "scc")
CODE_ID = {"cc": ecl.CC, "mis": ecl.MIS, "gc": ecl.GC, "mst": ecl.MST, "scc": ecl.SCC}
BATCH_ID = {"cc": ecl.BATCH_CC, "mis": ecl.BATCH_MIS, "gc": ecl.BATCH_GC, "mst": ecl.BATCH_MST, "scc": ecl.BATCH_SCC}


def listed():
    return [
        # the smallest calls: a thousand vertices, every code once -- launches
        # and latency, what a program pays that solves many tiny graphs singly
        dict(name="tiny-rmat10", kind="solve", codes="cc,mis,gc,mst,scc", family="rmat", n=1000, degree=8,
             symmetric=True, where="device", workspace=False),
        # the connected-components benchmark: a 1024 x 1024 grid, 5 % of edges deleted
        dict(name="cc-grid1024", kind="solve", codes="cc", family="grid", n=1024 * 1024, degree=2, symmetric=True,
             where="device", workspace=False),
        # the suite benchmark at R-MAT scale 22, edge factor 16, symmetrised:
        # the two codes that read the list once ...
        dict(name="cc-mis-rmat22", kind="solve", codes="cc,mis", family="rmat", n=1 << 22, degree=16, symmetric=True,
             where="device", workspace=False),
        # ... colouring (a long priority chain) ...
        dict(name="gc-rmat22", kind="solve", codes="gc", family="rmat", n=1 << 22, degree=16, symmetric=True,
             where="device", workspace=False),
        # ... spanning forest with weights ...
        dict(name="mst-rmat22", kind="solve", codes="mst", family="rmat", n=1 << 22, degree=16, symmetric=True,
             where="device", workspace=False),
        # ... and strongly connected components of the directed graph
        dict(name="scc-rmat22", kind="solve", codes="scc", family="rmat", n=1 << 22, degree=16, symmetric=False,
             where="device", workspace=False),
        # a mesh of ordinary, ragged size (no power of two, rows of at most
        # four entries), every code, with a workspace the program keeps
        dict(name="mesh-suite", kind="solve", codes="cc,mis,gc,mst,scc", family="grid", n=701 * 1031, degree=2,
             symmetric=True, where="device", workspace=True),
        # a graph in host memory, as the command-line tools and the
        # reference-shaped wrappers call the codes: copies in and out included
        dict(name="host-er", kind="solve", codes="cc,mis,gc,mst,scc", family="er", n=150001, degree=8, symmetric=True,
             where="host", workspace=False),
        # the all-pairs benchmark: n = 8192, edge probability 0.001
        dict(name="apsp-8192", kind="apsp", n=8192, degree=8),
        # an ordinary all-pairs call whose size is no multiple of any tile
        dict(name="apsp-1001", kind="apsp", n=1001, degree=12),
        # the batched benchmark's mix: CC, MIS and MST of many small graphs of
        # 1 k to 200 k vertices in one run, every result read back
        dict(name="batch-mix", kind="batch", codes="cc,mis,mst", graphs=96, n_min=1000, n_max=200000),
        # the served benchmark: a saturating Poisson stream of all codes over
        # resident R-MAT and grid graphs of 10 k vertices and more
        dict(name="serve-stream", kind="serve", graphs=10, n_min=10000, n_max=1 << 20, requests=50, rate=10000.0,
             slots=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.random()
    if what < 0.65:
        family = rng.choice(("rmat", "rmat", "grid", "er"))
        codes = ",".join(sorted(rng.sample(CODES, rng.choice((1, 1, 1, 2, 5))), key=CODES.index))
        host = rng.random() < 0.15
        n = _log_int(rng, 500, 1 << (19 if host else 22))
        return dict(kind="solve", codes=codes, family=family, n=n, degree=2 if family == "grid" else rng.randint(4, 16),
                    symmetric=codes not in ("cc", "scc") or rng.random() < (0.7 if codes == "cc" else 0.2), where="host" if host else "device",
                    workspace=rng.random() < 0.3)
    if what < 0.8:
        return dict(kind="apsp", n=_log_int(rng, 100, 6000), degree=rng.randint(4, 24))
    if what < 0.9:
        codes = ",".join(sorted(rng.sample(CODES, rng.randint(1, 3)), key=CODES.index))
        return dict(kind="batch", codes=codes, graphs=rng.randint(8, 96), n_min=1000, n_max=_log_int(rng, 5000, 200000))
    return dict(kind="serve", graphs=rng.randint(4, 10), n_min=10000, n_max=_log_int(rng, 50000, 1 << 20),
                requests=rng.randint(10, 50), rate=float(_log_int(rng, 5000, 10000)), slots=rng.choice((4, 8)))


# ---- graphs -----------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _csr(keys, n):
    """Sorted unique keys u * n + v -> (nindex, nlist), int32."""
    u = torch.div(keys, n, rounding_mode="floor")
    nindex = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(u, minlength=n), 0, out=nindex[1:])
    return nindex.to(torch.int32), (keys - u * n).to(torch.int32)


def _pair_weights(keys, n, seed, weight_max):
    """Weights uniform in [1, weight_max), equal for (u, v) and (v, u)."""
    u = torch.div(keys, n, rounding_mode="floor")
    v = keys - u * n
    x = torch.minimum(u, v) * n + torch.maximum(u, v) + seed * 0x1E3779B97F4A7C15 % (1 << 62)
    for _ in range(2):
        x = (x ^ ((x >> 29) & 0x7FFFFFFFF)) * 0x1F58476D1CE4E5B9
    x = (x >> 20) & 0x7FFFFFFFFFF
    return (1 + x % (weight_max - 1)).to(torch.int32)


def _edges(family, n, degree, seed):
    """(u, v) int64 samples of the family; duplicates and self-loops still in."""
    g = _gen(seed)
    if family == "grid":
        cols = max(1, int(round(math.sqrt(n))))
        while cols > 1 and n % cols and cols > math.sqrt(n) / 2:  # whole rows where n allows
            cols -= 1
        v = torch.arange(n, device="cuda")
        right = v[(v % cols != cols - 1) & (v + 1 < n)]
        down = v[v + cols < n]
        a = torch.cat((right, down))
        b = torch.cat((right + 1, down + cols))
        keep = torch.rand(a.numel(), generator=g, device="cuda") >= 0.05
        return a[keep], b[keep]
    if family == "er":
        e = max(1, n * degree // 2)
        return (torch.randint(n, (e,), generator=g, device="cuda"), torch.randint(n, (e,), generator=g, device="cuda"))
    scale = max(1, math.ceil(math.log2(n)))
    e = n * degree
    u = torch.zeros(e, dtype=torch.int32, device="cuda")
    v = torch.zeros(e, dtype=torch.int32, device="cuda")
    for _ in range(scale):  # quadrants .57 / .19 / .19 / .05
        r = torch.rand(e, generator=g, device="cuda")
        lower = r >= 0.76
        u.mul_(2).add_(lower)
        v.mul_(2).add_(((r >= 0.57) & ~lower) | (r >= 0.95))
    if n < 1 << scale:
        keep = (u < n) & (v < n)
        u, v = u[keep], v[keep]
    return u.to(torch.int64), v.to(torch.int64)


def _graph(family, n, degree, symmetric, seed, weight_max=WEIGHT_MAX):
    """A weighted DeviceGraph without self-loops or duplicates, lists sorted."""
    u, v = _edges(family, n, degree, seed)
    keep = u != v
    u, v = u[keep], v[keep]
    keys = torch.cat((u * n + v, v * n + u)) if symmetric else u * n + v
    del u, v, keep
    keys = torch.unique(keys)
    nindex, nlist = _csr(keys, n)
    weights = _pair_weights(keys, n, seed, weight_max)
    if not nlist.numel():
        nlist, weights = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.ones(1, dtype=torch.int32, device="cuda")
    return ecl.DeviceGraph(nindex, nlist, weights, symmetric, int(keys.numel()))


def _most_entries(family, n, degree, symmetric):
    """Entries the family's graph has at most, whatever the seed: MST flag
    buffers are this long (zeros past the graph's own entries)."""
    return max(1, 4 * n if family == "grid" else (2 if symmetric and family == "rmat" else 1) * n * degree)


def _to_host(g):
    return ecl.Graph(g.nindex.cpu().numpy(), g.nlist.cpu().numpy()[: g.edges], g.eweight.cpu().numpy()[: g.edges],
                     g.symmetric)


def _apsp_graph(case, seed):
    """Directed graph, weights uniform in [1, 1000] per entry."""
    n = case["n"]
    g = _gen(seed)
    e = max(1, n * case["degree"])
    u = torch.randint(n, (e,), generator=g, device="cuda")
    v = torch.randint(n, (e,), generator=g, device="cuda")
    keys = torch.unique((u * n + v)[u != v])
    nindex, nlist = _csr(keys, n)
    weights = torch.randint(1, 1001, (keys.numel(),), generator=g, device="cuda", dtype=torch.int32)
    return ecl.DeviceGraph(nindex, nlist, weights, False, int(keys.numel()))


def _spread(case, i):
    """Size of the i-th of a case's graphs: spread evenly over its range's logarithm, made odd."""
    x = math.log(case["n_min"]) + (i * 0.6180339887498949) % 1.0 * (math.log(case["n_max"]) - math.log(case["n_min"]))
    return int(math.exp(x)) | 1


# ---- one state, one pass ------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "apsp":
        return dict(kind=kind, graph=_apsp_graph(case, seed))
    if kind == "solve":
        g = _graph(case["family"], case["n"], case["degree"], case["symmetric"], seed)
        codes = case["codes"].split(",")
        keep = {}
        if case["workspace"]:  # a program that calls often keeps one workspace for all its calls
            size = max(ecl.workspace_bytes(CODE_ID[c], g.nodes, g.edges) for c in codes)
            keep["workspace"] = torch.empty(size + 1024, dtype=torch.uint8, device="cuda")
        flags = None
        if "mst" in codes:
            flags = torch.zeros(_most_entries(case["family"], case["n"], case["degree"], case["symmetric"]),
                                dtype=torch.uint8, device="cuda")
        if case["where"] == "host":
            g, flags = _to_host(g), None if flags is None else flags.cpu().numpy()
        return dict(kind=kind, graph=g, codes=codes, keep=keep, flags=flags)
    if kind == "batch":
        # every result goes to its place in one page-locked buffer a code, as a
        # program does that hands the results of a whole batch on
        codes = case["codes"].split(",")
        b = ecl.Batch()
        outs = {c: [] for c in codes}
        for i in range(case["graphs"]):
            family, n = ("er", "grid", "rmat")[i % 3], _spread(case, i)
            b.add(_to_host(_graph(family, n, 8, True, seed * 1000 + i, 1 << 16)))
            for c in codes:
                outs[c].append(_most_entries(family, n, 8, True) if c == "mst" else n)
        b.build(sum(BATCH_ID[c] for c in codes))
        places = []
        for c in codes:
            flat = torch.zeros(sum(outs[c]), dtype=torch.uint8 if c in ("mis", "mst") else torch.int32).pin_memory()
            at = flat.data_ptr()
            for i, k in enumerate(outs[c]):
                places.append((i, BATCH_ID[c], at))
                at += k * flat.element_size()
            outs[c] = flat
        return dict(kind=kind, batch=b, places=places, outs=outs)
    srv = ecl.Server(slots=case["slots"])
    rng = np.random.default_rng(seed)
    graphs = []
    for i in range(case["graphs"]):
        family, n = "rmat" if i % 2 else "grid", _spread(case, i)
        gid = srv.add_graph(_to_host(_graph(family, n, 8 + i % 9, True, seed * 1000 + i)))
        graphs.append((gid, n, _most_entries(family, n, 8 + i % 9, True)))
    requests, outs, at = [], [], 0.0
    for r in range(case["requests"]):
        gid, n, most = graphs[r % len(graphs)]
        code = CODES[(r + r // len(CODES)) % len(CODES)]
        at += float(rng.exponential(1.0 / case["rate"]))
        out = torch.zeros(most if code == "mst" else n, dtype=torch.uint8 if code in ("mis", "mst") else torch.int32)
        out = out.pin_memory()
        outs.append(out)
        requests.append((CODE_ID[code], gid, at, out.data_ptr()))
    return dict(kind=kind, server=srv, requests=requests, outs=outs)


def run(state):
    kind = state["kind"]
    if kind == "apsp":
        return ecl.apsp(state["graph"])
    if kind == "solve":
        results = []
        for c in state["codes"]:
            if c == "mst":
                _, total = ecl.mst(state["graph"], out=state["flags"], **state["keep"])
                results += [state["flags"], total]
            else:
                results.append(getattr(ecl, c)(state["graph"], **state["keep"]))
        return results
    if kind == "batch":
        b = state["batch"]
        b.run()
        totals = np.zeros(b.graphs, dtype=np.uint64)
        failed = 0
        for i, code, at in state["places"]:
            total = totals[i : i + 1].ctypes.data_as(C.POINTER(C.c_uint64)) if code == ecl.BATCH_MST else None
            failed += ecl.lib.ecl_batch_result(b.h, i, code, at, total) != ecl.OK
        return [failed, totals.astype(np.int64), state["outs"]]
    status, done, _ = state["server"].run(state["requests"])
    return [status, np.array([r.status for r in done]), np.array([r.total_weight for r in done], dtype=np.int64),
            state["outs"]]


# ---- what a pass cannot do without ----------------------------------------------------


def _entries(family, n, degree, symmetric):
    """About the CSR entries of such a graph (duplicates of R-MAT samples leave it)."""
    if family == "grid":
        return 3.8 * n
    if family == "er":
        return float(degree * n)
    return (1.9 if symmetric else 0.95) * degree * n


def _solve_bytes(code, n, m):
    """The CSR (and weights) read once, the result written once."""
    if code == "mst":
        return 4 * n + 8 * m + m
    return 4 * n + 4 * m + (n if code == "mis" else 4 * n)


def work(case):
    kind = case["kind"]
    if kind == "apsp":
        n = float(case["n"])
        return {"bytes": 4 * n * n + 8 * n * case["degree"], "flops": 2 * n ** 3}
    total = 0.0
    if kind == "solve":
        n = case["n"]
        m = _entries(case["family"], n, case["degree"], case["symmetric"])
        total = sum(_solve_bytes(c, n, m) for c in case["codes"].split(","))
    elif kind == "batch":
        for i in range(case["graphs"]):
            n = _spread(case, i)
            m = _entries(("er", "grid", "rmat")[i % 3], n, 8, True)
            total += sum(_solve_bytes(c, n, m) for c in case["codes"].split(","))
    else:
        for r in range(case["requests"]):
            i = r % case["graphs"]
            n = _spread(case, i)
            m = _entries("rmat" if i % 2 else "grid", n, 8 + i % 9, True)
            total += _solve_bytes(CODES[(r + r // len(CODES)) % len(CODES)], n, m)
    return {"bytes": total, "flops": 0.0}


def exact(case, seed):
    """All-pairs distances in 64 bits by plain Floyd-Warshall; the other codes
    return ids, flags and colours."""
    if case["kind"] != "apsp":
        return None
    g = _apsp_graph(case, seed)
    n = case["n"]
    d = torch.full((n, n), ecl.APSP_INF, dtype=torch.int64, device="cuda")
    d.fill_diagonal_(0)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (g.nindex[1:] - g.nindex[:-1]).to(torch.int64))
    d[rows, g.nlist.to(torch.int64)] = g.eweight.to(torch.int64)
    for k in range(n):
        torch.minimum(d, d[:, k : k + 1] + d[k : k + 1, :], out=d)
    return d
