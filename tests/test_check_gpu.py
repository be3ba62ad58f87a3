"""The device checker (pbg_bfs_check, pbg_levels_check) against the oracle's
restatement of checkBFS (BFSCheck.C:39-90).  Mistakes are planted in host
copies of parent arrays and level rows; the verdict (first bad vertex, or
none) must be the oracle's."""
import numpy as np
import pytest
import torch

import pbbsbench_b200 as pb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NONE = pb.NONE


def _gpu_verdict(dg, src, parent, edges=True):
    d = torch.from_numpy(np.ascontiguousarray(parent).view(np.int32)).cuda()
    r = dg.check(src, d, edges=edges)
    return r["bad_vertex"]


def _oracle_verdict(off, edg, src, parent, edges=True):
    b = O.check_bfs(off, edg, src, np.ascontiguousarray(parent).view(np.uint32), check_edges=edges)
    return NONE if b < 0 else b


@pytest.fixture(scope="module")
def graph():
    off, edg = O.rmat(14, 10 << 14, 21, 0.5, 0.1, 0.1)
    return off, edg


def test_valid_trees(cuda_device, graph):
    off, edg = graph
    dg = pb.DeviceGraph.upload(off, edg)
    for src in (0, 5, 999):
        for mode in (pb.PARENT_ANY, pb.PARENT_MIN, pb.PARENT_MAX):
            par, _, _ = dg.bfs(src, parent_mode=mode)
            assert _gpu_verdict(dg, src, par) == NONE
    dg.close()


def test_planted_mistakes(cuda_device, graph):
    off, edg = graph
    dg = pb.DeviceGraph.upload(off, edg)
    src = 0
    par, lv, _ = dg.bfs(src, levels=True)
    par = par.view(np.uint32).copy()
    lv = lv.copy()
    reached = np.nonzero((lv != NONE) & (np.arange(len(lv)) != src))[0]
    rng = np.random.default_rng(3)
    deep = reached[np.argsort(lv[reached])][-50:]
    cases = {}
    p = par.copy(); p[src] = int(deep[0]); cases["start not its own parent"] = p
    v = int(deep[-1]); p = par.copy(); p[v] = par[par[v]]; cases["parent two levels up"] = p
    v = int(deep[-2]); same = np.nonzero(lv == lv[par[v]])[0]
    nbrs = set(edg[off[v]:off[v + 1]].tolist())
    cand = [int(u) for u in same if int(u) not in nbrs]
    p = par.copy(); p[v] = cand[0]; cases["parent not a neighbour"] = p
    v = int(deep[-3]); p = par.copy(); p[v] = NONE; cases["reached reported unreached"] = p
    un = np.nonzero(lv == NONE)[0]
    if len(un):
        p = par.copy(); p[int(un[0])] = src; cases["unreached given a parent"] = p
    a, b = int(deep[-4]), int(deep[-5]); p = par.copy(); p[a] = b; p[b] = a; cases["cycle"] = p
    p = par.copy(); p[int(deep[-6])] = len(lv) + 7; cases["parent not a vertex"] = p
    for name, p in cases.items():
        for edges in (True, False):
            want = _oracle_verdict(off, edg, src, p, edges)
            got = _gpu_verdict(dg, src, p, edges)
            assert got == want, (name, edges, got, want)
            # only the edge test sees a non-neighbour parent at the right level
            if name != "parent not a neighbour" or edges:
                assert want != NONE, (name, edges)
    dg.close()


def test_levels_rows(cuda_device, graph):
    off, edg = graph
    dg = pb.DeviceGraph.upload(off, edg)
    n = dg.n
    srcs = np.array([0, 7, 123, 4096], np.uint32)
    lv, _ = dg.bfs_multi(srcs)
    d = torch.from_numpy(lv.reshape(-1)).cuda()
    assert dg.levels_check(srcs, d)["bad_vertex"] == NONE
    bad = lv.copy()
    v = int(np.nonzero(bad[2] == 3)[0][0])
    bad[2, v] = 5
    r = dg.levels_check(srcs, torch.from_numpy(bad.reshape(-1)).cuda())
    assert r["row"] == 2 and r["bad_vertex"] <= v
    bad = lv.copy()
    bad[1, srcs[1]] = 1
    r = dg.levels_check(srcs, torch.from_numpy(bad.reshape(-1)).cuda())
    assert r["row"] == 1 and r["bad_vertex"] <= srcs[1]
    dg.close()


def test_full_size_rmat24_tree(cuda_device):
    """The C3 graph: a parent tree from the device search checked on the
    device in well under a second."""
    dg = pb.rmat_graph(24, 1 << 28, 3, 0.57, 0.19, 0.19)
    off = dg.download_offsets()
    src = int(np.nonzero(np.diff(off))[0][0])
    par = torch.empty(dg.n, dtype=torch.int32, device="cuda")
    dg.bfs_device(src, par)
    torch.cuda.synchronize()
    assert dg.check(src, par)["bad_vertex"] == NONE
    dg.close()


def test_long_lists_checked_through_their_tails(cuda_device):
    """A vertex whose list is longer than the 64 entries one lane scans: its
    only neighbour one level up (its parent) sits in the list's tail, which
    the device check reads in pieces spread over the grid.  A correct tree
    passes only if the tail's minimum level and adjacency are used; a parent
    at the right level that is not a neighbour is caught by the edge test."""
    n, h, p, q = 1000, 999, 900, 950
    us = [0, p, 0] + [h] * 399
    vs = [p, h, q] + list(range(1, 400))
    off, edg = O.csr_symmetric(n, np.array(us, np.uint32), np.array(vs, np.uint32))
    assert off[h + 1] - off[h] == 400 and list(edg[off[h]:off[h + 1]]).index(p) == 399
    dg = pb.DeviceGraph.upload(off, edg)
    par, lv, _ = dg.bfs(0, levels=True)
    par = par.view(np.uint32).copy()
    assert par[h] == p and lv[h] == 2
    cases = {"valid": par}
    x = par.copy(); x[h] = q; cases["parent at the right level, not a neighbour"] = x
    x = par.copy(); x[p] = NONE; cases["the tail neighbour unreached"] = x
    for name, pp in cases.items():
        for edges in (True, False):
            want = _oracle_verdict(off, edg, 0, pp, edges)
            got = _gpu_verdict(dg, 0, pp, edges)
            assert got == want, (name, edges, got, want)
    assert _oracle_verdict(off, edg, 0, par, True) == NONE
    assert _oracle_verdict(off, edg, 0, cases["parent at the right level, not a neighbour"], True) == h
    assert _oracle_verdict(off, edg, 0, cases["parent at the right level, not a neighbour"], False) == NONE
    dg.close()


def _levels_verdict(off, edg, srcs, rows):
    """First failing (row, vertex) of the level predicate with its level and lowest neighbour level, in numpy."""
    n = len(off) - 1
    deg = np.diff(off).astype(np.int64)
    for r in range(len(srcs)):
        lv = rows[r].astype(np.int64)
        lv[lv == 255] = n
        mn = np.full(n, n, np.int64)
        np.minimum.at(mn, np.repeat(np.arange(n), deg), lv[edg])
        ok = ((lv == n) & (mn == n)) | ((mn < n) & (lv == mn + 1))
        ok[srcs[r]] = lv[srcs[r]] == 0
        if not ok.all():
            v = int(np.argmin(ok))
            return {"bad_vertex": v, "row": r, "level": int(lv[v]), "min_neighbor_level": int(mn[v])}
    return None


@pytest.mark.parametrize("n", [200, 257, 4099])
@pytest.mark.parametrize("k", [1, 4, 5, 17, 33, 64, 67])
def test_levels_rows_in_strips(cuda_device, n, k):
    """Row counts on both sides of every strip width, an odd n, lists of over 64 and over 320 entries (one and several
    tail pieces), unreached vertices, and faults whose only evidence is in a list's tail."""
    rng = np.random.default_rng(n * 100 + k)
    us, vs = [], []
    for hub, d in ((0, min(n - 9, 900)), (1, min(n - 9, 90))):
        to = rng.choice(np.arange(2, n - 6), d - 2, replace=False)
        us += [hub] * len(to)
        vs += to.tolist()
    a, b = rng.integers(2, n - 6, 3 * n), rng.integers(2, n - 6, 3 * n)
    off, edg = O.csr_symmetric(n, np.array(us + a.tolist(), np.uint32), np.array(vs + b.tolist(), np.uint32))
    dg = pb.DeviceGraph.upload(off, edg)
    srcs = rng.choice(np.nonzero(np.diff(off))[0], k).astype(np.uint32)
    srcs[0] = 0
    rows = np.stack([np.minimum(O.bfs_levels(off, edg, int(s)).astype(np.int64), 255).astype(np.uint8) for s in srcs])

    def both(x):
        got = dg.levels_check(srcs, torch.from_numpy(x.reshape(-1)).cuda())
        want = _levels_verdict(off, edg, srcs, x)
        if want is None:
            assert got["bad_vertex"] == NONE
        else:
            assert got == want
        return want

    assert both(rows) is None
    for r in sorted({0, k // 2, k - 1}):
        for v, to in ((int(srcs[r]), 1), (int(edg[off[1] - 1]), 3), (n - 1, 7), (int(edg[off[1] - 1]), 255),
                      (int(edg[off[2] - 1]), 0), (int(rng.integers(0, n)), 254), (2, n if n < 255 else 254)):
            bad = rows.copy()
            bad[r, v] = to if bad[r, v] != to else to ^ 1
            assert both(bad) is not None or n < 255
    dg.close()


class _Hog:
    """Takes all device memory but `left` bytes."""

    def __init__(self, left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(max(0, free - left) >> 21 << 21, dtype=torch.uint8, device="cuda")
        now, _ = torch.cuda.mem_get_info()
        assert abs(now - left) <= 4 << 20, (free, now, left)

    def release(self):
        self.block = None
        torch.cuda.empty_cache()


@pytest.fixture
def hog(cuda_device):
    held = []

    def take(left):
        held.append(_Hog(left))

    yield take
    for h in held:
        h.release()


def _warm_levels_check():
    """Every width's kernels once: a kernel is loaded into device memory when it is first launched."""
    off, edg = O.csr_symmetric(700, np.zeros(600, np.uint32), np.arange(1, 601, dtype=np.uint32))
    for cut, ks in ((700, (2, 12, 20, 40)), (200, (2,))):
        o = np.minimum(off[: cut + 1], 0) if cut < 700 else off
        dg = pb.DeviceGraph.upload(o, edg[: o[-1]])
        for k in ks:
            rows = np.full((k, cut), 255, np.uint8)
            dg.levels_check(np.zeros(k, np.uint32), torch.from_numpy(rows).cuda())
        dg.close()


def test_level_rows_without_memory_for_the_tail_table(hog):
    """Lists of 40,000 entries (every neighbour twenty times over): the table of their tails takes 10 MB.  With less
    than that left the rows are checked all the same."""
    n, reach, times = 4096, 1000, 20
    d = torch.arange(1, reach + 1, dtype=torch.int32, device="cuda")
    to = torch.cat([d, -d]).repeat_interleave(times)
    edges = (torch.arange(n, dtype=torch.int32, device="cuda")[:, None] + to[None, :]).remainder_(n).reshape(-1)
    off = torch.arange(n + 1, dtype=torch.int64, device="cuda").mul_(2 * reach * times).to(torch.int32)
    dg = pb.DeviceGraph.upload(off, edges)
    del edges, to
    srcs = np.array([0, 1777], np.uint32)
    gap = np.abs(np.arange(n)[None, :] - srcs[:, None])
    rows = (-(-np.minimum(gap, n - gap) // reach)).astype(np.uint8)
    bad = rows.copy()
    bad[1, 3000] += 1
    d_rows, d_bad = torch.from_numpy(rows).cuda(), torch.from_numpy(bad).cuda()
    _warm_levels_check()
    hog(6 << 20)
    assert dg.levels_check(srcs, d_rows)["bad_vertex"] == NONE
    got = dg.levels_check(srcs, d_bad)
    assert got["row"] == 1 and got["bad_vertex"] <= 3000
    dg.close()


@pytest.mark.parametrize("left", [250, 150, 100, 40])
def test_level_rows_in_narrower_strips(hog, left):
    """40 rows of 4.1 M vertices take 328 MB of scratch in strips of 64; with 250, 150, 100 and 40 MB left they go
    through strips of 32, 16 and 4 rows, and row by row."""
    k = 40
    make = lambda: pb.torus3d_graph(160, perm_seed=3)  # noqa: E731
    with_levels = make()
    srcs = np.arange(5, 5 + 1000 * k, 1000, dtype=np.uint32)
    rows, _ = with_levels.bfs_multi(srcs)
    with_levels.close()
    dg = make()
    d_rows = torch.from_numpy(rows).cuda()
    v = int(np.argmax(rows[33]))
    _warm_levels_check()
    hog(left << 20)
    assert dg.levels_check(srcs, d_rows)["bad_vertex"] == NONE
    d_rows[33, v] += 1
    got = dg.levels_check(srcs, d_rows)
    assert got["row"] == 33 and got["bad_vertex"] <= v
    dg.close()
