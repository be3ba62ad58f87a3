"""The work that programs have this library do, as cases that can be timed and compared.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (a resident graph,
output buffers, a batch object), ``run`` makes one pass through the public entry points.  Graphs are the kinds that
the library generates (rMat, 3-D torus, random-local) and directed graphs uploaded from device arrays.

Searches with the ANY parent rule return their levels only: which of a vertex's possible parents claims it first is not
determined, two runs differ.  The MIN and MAX rules return parents too.  All outputs are whole numbers.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import pbbsbench_b200 as pb

DEV = "cuda"
MODES = {"any": pb.PARENT_ANY, "min": pb.PARENT_MIN, "max": pb.PARENT_MAX}


def listed():
    return [
        # the smallest call: one search on a graph of a few thousand vertices, where launches and barriers are all there is
        dict(name="bfs_rmat12", op="bfs", graph="rmat", logn=12, per=16, mode="any"),
        # the plugin's call: deterministic parents and distances as host arrays, social-network-like graph of a million vertices
        dict(name="bfs_host_rmat20_min", op="bfs_host", graph="rmat", logn=20, per=10, mode="min"),
        # high diameter, 240 levels of small frontiers: a lattice with ids in random order
        dict(name="bfs_torus160", op="bfs", graph="torus", dn=160, mode="any"),
        # the headline: direction-optimizing search on 2^24 vertices and half a billion edges
        dict(name="bfs_rmat24", op="bfs", graph="rmat", logn=24, per=16, mode="any"),
        # directed graph (top-down only), odd size, skewed degrees, the deterministic max-parent rule
        dict(name="bfs_directed_max", op="bfs", graph="directed", n=2000003, degree=12, mode="max"),
        # one batched job of 64 sources on a graph with many levels
        dict(name="ms64_randlocal23", op="multi", graph="randlocal", n=1 << 23, degree=5, window=1 << 16, k=64),
        # the served shape: eight graphs of uneven sizes, 64 sources each, one fused launch
        dict(name="ms64_fused_rmat16_23", op="fused", lo=16, hi=23, per=16, k=64),
        # the widest job: 256 sources
        dict(name="ms256_rmat20", op="multi", graph="rmat", logn=20, per=16, k=256),
        # maximal independent set on the headline graph
        dict(name="mis_rmat24", op="mis", graph="rmat", logn=24, per=16),
        # construction of the headline graph: draws to a validated, symmetric, resident CSR
        dict(name="build_rmat24", op="build", graph="rmat", logn=24, per=16),
        # an AdjacencyGraph text in host memory to a resident graph, symmetry found by the library (its default)
        dict(name="load_text_rmat20", op="load", graph="rmat", logn=20, per=10),
        # the checker: a search's parents and a batch's 64 level rows, right ones and ones with a planted fault
        dict(name="verify_rmat20", op="verify", graph="rmat", logn=20, per=16, k=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, max_edges):
    """A graph of a random kind and size with at most about max_edges directed edges."""
    kind = rng.choice(["rmat", "rmat", "torus", "randlocal"])
    if kind == "rmat":
        per = rng.randint(6, 20)
        top = min(24, int(math.log2(max_edges / (2 * per))))
        return dict(graph="rmat", logn=rng.randint(10, top), per=per)
    if kind == "torus":
        return dict(graph="torus", dn=_log_int(rng, 11, min(160, int((max_edges / 6) ** (1 / 3)))))
    degree = rng.randint(3, 8)
    n = _log_int(rng, 3001, min(1 << 23, max_edges // (2 * degree)))
    return dict(graph="randlocal", n=n, degree=degree, window=max(16, int(n * rng.uniform(0.008, 0.05))))


def draw(rng):
    op = rng.choice(["bfs", "bfs", "bfs_host", "bfs_directed", "multi", "multi_wide", "fused", "mis", "build", "load",
                     "verify"])
    if op == "bfs":
        return dict(op="bfs", mode=rng.choice(["any", "min", "max"]), **_draw_graph(rng, 500_000_000))
    if op == "bfs_host":
        return dict(op="bfs_host", mode=rng.choice(["min", "max"]), **_draw_graph(rng, 40_000_000))
    if op == "bfs_directed":
        return dict(op="bfs", graph="directed", n=_log_int(rng, 5001, 4_000_001), degree=rng.randint(4, 24),
                    mode=rng.choice(["any", "min", "max"]))
    if op == "multi":
        g = _draw_graph(rng, 60_000_000)
        while g["graph"] == "torus" and g["dn"] > 80:  # the levels of a batch fit a byte
            g = _draw_graph(rng, 60_000_000)
        return dict(op="multi", k=rng.randint(1, 64), **g)
    if op == "multi_wide":
        g = _draw_graph(rng, 16_000_000)
        while g["graph"] == "torus" and g["dn"] > 80:
            g = _draw_graph(rng, 16_000_000)
        return dict(op="multi", k=rng.randint(65, 256), **g)
    if op == "fused":
        lo = rng.randint(10, 16)
        return dict(op="fused", lo=lo, hi=rng.randint(lo + 1, 21), per=rng.randint(8, 16), k=rng.randint(16, 64))
    if op == "mis":
        return dict(op="mis", **_draw_graph(rng, 500_000_000))
    if op == "build":
        return dict(op="build", **_draw_graph(rng, 400_000_000))
    if op == "load":
        return dict(op="load", **_draw_graph(rng, 20_000_000))
    g = _draw_graph(rng, 30_000_000)
    while g["graph"] == "torus" and g["dn"] > 80:
        g = _draw_graph(rng, 30_000_000)
    return dict(op="verify", k=rng.randint(1, 64), **g)


class _View:
    """A device array of a graph handle, for torch, which keeps the handle alive as long as its tensors."""

    def __init__(self, graph, ptr, count):
        self.graph = graph
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (int(count),), "typestr": "<i4", "version": 2}


def _csr(g):
    """The resident offsets and edges as torch tensors."""
    arrays = (g.d_offsets, g.n + 1), (g.d_edges, max(1, g.m))  # every allocation holds a few words at least
    off, edges = (torch.as_tensor(_View(g, ptr, count), device=DEV) for ptr, count in arrays)
    return off, edges[: g.m]


def _graph(g, case):
    """The whole graph as arrays whose sizes do not depend on how many duplicate edges the seed gave: offsets, and the
    first and the last edges, each half of what there is without duplicates (at most half of them are duplicates)."""
    off, edges = _csr(g)
    half = (_drawn_edges(case) + 1) // 2
    return off, edges[:half], edges[max(0, g.m - half):]


def _make(case, seed):
    kind = case["graph"]
    if kind == "rmat":
        return pb.rmat_graph(case["logn"], case["per"] << case["logn"], seed, 0.57, 0.19, 0.19)
    if kind == "torus":
        return pb.torus3d_graph(case["dn"], perm_seed=seed)
    if kind == "randlocal":
        return pb.randlocal_graph(case["n"], case["degree"], case["window"], seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n = case["n"]
    # a tenth of the vertices have ten times the out-degree of the others, and low ids are more often targets
    deg = torch.randint(0, case["degree"] + 1, (n,), generator=gen, device=DEV)
    deg = torch.where(torch.rand(n, generator=gen, device=DEV) < 0.1, deg * 10, deg)
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(deg, 0)
    m = int(off[-1])
    edges = (torch.rand(m, generator=gen, device=DEV, dtype=torch.float64) ** 2 * n).to(torch.int32)
    return pb.DeviceGraph.upload(off.to(torch.int32), edges, symmetric=False)


def _sources(g, k, seed):
    """k distinct vertices with out-edges (fewer where the graph has fewer), as host ids."""
    off, _ = _csr(g)
    live = torch.nonzero(off[1:] != off[:-1]).flatten()
    gen = torch.Generator(device=DEV).manual_seed(seed ^ 0x5EED)
    if k == 1:
        return live[torch.randint(0, live.numel(), (1,), generator=gen, device=DEV)].cpu().numpy().astype(np.uint32)
    at = torch.randint(0, live.numel(), (4 * k,), generator=gen, device=DEV)
    ids = list(dict.fromkeys(live[at].tolist()))[:k]
    return np.array(ids, dtype=np.uint32)


def _job(g, k, seed):
    srcs = _sources(g, k, seed)
    return pb.MultiWorkspace(g, max_sources=k), srcs, torch.empty((len(srcs), g.n), dtype=torch.uint8, device=DEV)


def prepare(case, seed):
    op = case["op"]
    s = dict(op=op)
    if op in ("build", "load"):
        s["case"] = dict(case)
    if op == "build":
        s["seed"] = seed
        return s
    if op == "fused":
        graphs = [_make(dict(graph="rmat", logn=lg, per=case["per"]), seed + lg) for lg in range(case["lo"], case["hi"] + 1)]
        s.update(graphs=graphs, jobs=[_job(g, case["k"], seed + i) for i, g in enumerate(graphs)],
                 batch=pb.Batch(len(graphs)))
        return s
    g = _make(case, seed)
    if op == "load":
        fd, path = tempfile.mkstemp(suffix=".adj")
        os.close(fd)
        try:
            g.write_adjacency(path)
            with open(path, "rb") as f:
                s["text"] = f.read()
        finally:
            os.unlink(path)
        g.close()
        return s
    s["g"] = g
    if op in ("bfs", "bfs_host"):
        s.update(src=int(_sources(g, 1, seed)[0]), mode=MODES[case["mode"]])
        if op == "bfs":
            s.update(parent=torch.empty(g.n, dtype=torch.int32, device=DEV), level=torch.empty(g.n, dtype=torch.int32, device=DEV))
    elif op == "mis":
        s["flags"] = torch.empty(g.n, dtype=torch.uint8, device=DEV)
    elif op == "multi":
        s.update(jobs=[_job(g, case["k"], seed)], batch=pb.Batch(1))
    elif op == "verify":
        _prepare_verify(s, case, seed)
    return s


def _prepare_verify(s, case, seed):
    """A search's parents and a batch's level rows, and copies of both with one fault."""
    g = s["g"]
    gen = torch.Generator(device=DEV).manual_seed(seed ^ 0xFA17)

    def pick(mask):
        at = torch.nonzero(mask).flatten()
        return int(at[torch.randint(0, at.numel(), (1,), generator=gen, device=DEV)]) if at.numel() else None

    ws, srcs, rows = _job(g, case["k"], seed)
    batch = pb.Batch(1)
    batch.launch([(ws, srcs, rows)])
    src = int(srcs[0])
    parent = torch.empty(g.n, dtype=torch.int32, device=DEV)
    level = torch.empty(g.n, dtype=torch.int32, device=DEV)
    g.bfs_device(src, parent, level, parent_mode=pb.PARENT_MIN)
    torch.cuda.synchronize()
    # a parent one level up that is (most likely) no neighbour
    bad_parent = parent.clone()
    v = pick((level >= 2) & (level < g.n))
    if v is not None:
        bad_parent[v] = pick(level == level[v] - 1)
    # a vertex of a row's last level, one too deep
    bad_rows = rows.clone()
    r = int(torch.randint(0, len(srcs), (1,), generator=gen, device=DEV))
    row = bad_rows[r]
    last = int(torch.where(row == 255, torch.zeros_like(row), row).max())
    v = pick(row == last)
    row[v] = last + 1
    ws.close()
    batch.close()
    s.update(srcs=srcs, src=src, parent=parent, rows=rows, bad_parent=bad_parent, bad_rows=bad_rows)


def run(s):
    op = s["op"]
    if op == "bfs":
        s["g"].bfs_device(s["src"], s["parent"], s["level"], parent_mode=s["mode"])
        return s["level"] if s["mode"] == pb.PARENT_ANY else (s["parent"], s["level"])
    if op == "bfs_host":
        parent, level, _ = s["g"].bfs(s["src"], parent_mode=s["mode"], levels=True)
        return parent, level.view(np.int32)
    if op in ("multi", "fused"):
        s["batch"].launch(s["jobs"])
        return [rows for _, _, rows in s["jobs"]]
    if op == "mis":
        s["g"].mis_device(s["flags"])
        return s["flags"]
    if op == "build":
        s["g"] = None  # the graph of the pass before is given back first
        s["g"] = _make(s["case"], s["seed"])
        return _graph(s["g"], s["case"])
    if op == "load":
        s["g"] = None
        s["g"] = pb.DeviceGraph.parse_adjacency(s["text"])
        flags = ctypes.c_uint32()
        pb.lib().pbg_graph_flags(s["g"].handle, ctypes.byref(flags))
        return *_graph(s["g"], s["case"]), flags.value
    g = s["g"]
    return [g.check(s["src"], s["parent"]), g.check(s["src"], s["bad_parent"]),
            g.levels_check(s["srcs"], s["rows"]), g.levels_check(s["srcs"], s["bad_rows"])]


def _drawn_edges(case):
    """Directed edges of a generated graph before duplicates and self loops are dropped."""
    kind = case["graph"]
    if kind == "rmat":
        return 2 * (case["per"] << case["logn"])
    return 6 * case["dn"] ** 3 if kind == "torus" else 2 * case["degree"] * case["n"]


def _size(case):
    """(vertices, directed edges) of the case's graph, edges to a few per cent (duplicates are dropped)."""
    kind = case["graph"]
    if kind == "rmat":
        return 1 << case["logn"], int(0.97 * _drawn_edges(case))
    if kind == "torus":
        return case["dn"] ** 3, _drawn_edges(case)
    if kind == "randlocal":
        return case["n"], _drawn_edges(case)
    return case["n"], int(case["n"] * case["degree"] / 2 * 1.9)


def work(case):
    op = case["op"]
    if op == "fused":
        sizes = [_size(dict(graph="rmat", logn=lg, per=case["per"])) for lg in range(case["lo"], case["hi"] + 1)]
        return {"bytes": sum(4 * (n + 1) + 4 * m + case["k"] * n for n, m in sizes), "flops": 0}
    n, m = _size(case)
    csr = 4 * (n + 1) + 4 * m
    if op in ("bfs", "bfs_host"):
        return {"bytes": csr + 8 * n, "flops": 0}  # parents and levels written
    if op == "multi":
        return {"bytes": csr + case["k"] * n, "flops": 0}
    if op == "mis":
        return {"bytes": csr + n, "flops": 0}
    if op == "build":
        return {"bytes": csr, "flops": 0}  # made from a seed: only the result
    if op == "load":  # about digits + 1 characters a value
        return {"bytes": csr + m * (math.log10(n) + 0.9) + n * (math.log10(m) + 0.9), "flops": 0}
    return {"bytes": 2 * (csr + 4 * n) + 2 * (csr + case["k"] * n), "flops": 0}


def exact(case, seed):
    """All outputs are whole numbers: they are equal or they are wrong."""
    return None
