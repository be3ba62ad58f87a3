"""Graphs of the largest edge counts that a handle takes, 2^32 - 1, and that the
searches take, 64 less.

A list that ends there leaves no room in 32 bits for a cursor that steps past
its end.  65,536 vertices in pairs hold nearly all of the edges (each its
partner's id, over and over); the searched component's lists lie at the very
end, the last one short, one lane's share or a hub's.  The oracle sees the
same graph with each pair's list cut to one entry: sets, levels and verdicts
are the same.
"""
import numpy as np
import pytest
import torch

import pbbsbench_b200 as pb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

M = (1 << 32) - 1
M_SEARCH = M - 64
PAIRED = 1 << 16
TAIL = 600


class Case:
    """The graph on the device, and its short form on the host."""

    def __init__(self, hub, m):
        rng = np.random.default_rng(hub)
        last = TAIL - 1
        us = np.concatenate([rng.integers(0, last, 700), np.full(hub, last)])
        vs = np.concatenate([rng.integers(0, last, 700), rng.permutation(last)[:hub]])
        keep = us != vs
        toff, tedg = O.csr_symmetric(TAIL, us[keep].astype(np.uint32), vs[keep].astype(np.uint32))
        assert toff[-1] - toff[-2] == hub
        self.n = PAIRED + TAIL
        ids = np.arange(PAIRED, dtype=np.uint32)
        self.off = np.concatenate([ids, PAIRED + toff]).astype(np.uint32)
        self.edg = np.concatenate([ids ^ 1, PAIRED + tedg]).astype(np.uint32)
        filler = m - len(tedg)
        per, more = divmod(filler, PAIRED)
        lens = np.full(PAIRED, per, np.int64)
        lens[:more] += 1
        ends = np.cumsum(lens)
        off = np.concatenate([[0], ends, ends[-1] + toff[1:].astype(np.int64)]).astype(np.uint32)
        assert int(off[-1]) == m
        d_off = torch.from_numpy(off.view(np.int32)).cuda()
        d_edg = torch.empty(m, dtype=torch.int32, device="cuda")
        partner = torch.from_numpy((ids ^ 1).view(np.int32)).cuda()
        d_edg[: more * (per + 1)].view(more, per + 1)[:] = partner[:more, None]
        d_edg[more * (per + 1): filler].view(PAIRED - more, per)[:] = partner[more:, None]
        d_edg[filler:] = torch.from_numpy((PAIRED + tedg).astype(np.int32)).cuda()
        self.dg = pb.DeviceGraph.upload(d_off, d_edg)
        del d_edg
        torch.cuda.empty_cache()
        self.hub = PAIRED + last
        self.srcs = np.array([self.hub, PAIRED + tedg[-1], PAIRED + tedg[-2], PAIRED + 300], np.uint32)


@pytest.fixture(scope="module", params=[3, 40, 100, 300])
def case(cuda_device, request):
    c = Case(request.param, M)
    yield c
    c.dg.close()


@pytest.fixture(scope="module", params=[3, 31, 40, 300])
def searched(cuda_device, request):
    c = Case(request.param, M_SEARCH)
    yield c
    c.dg.close()


def test_independent_set(case):
    flags, st = case.dg.mis()
    want = O.mis_serial(case.off, case.edg)
    assert np.array_equal(flags, want) and st["in_set"] == int((want == 1).sum())


@pytest.mark.parametrize("rows", [2, 12, 20, 64])
def test_level_rows(case, rows):
    srcs = np.resize(case.srcs, rows)
    lv = np.ascontiguousarray(O.levels_u8(case.off, case.edg, srcs))
    assert case.dg.levels_check(srcs, torch.from_numpy(lv).cuda())["bad_vertex"] == pb.NONE
    assert lv[1, case.hub] == 1  # the last list's vertex, from a neighbour: one level too deep
    lv[1, case.hub] = 2
    r = case.dg.levels_check(srcs, torch.from_numpy(lv).cuda())
    assert r["row"] == 1 and r["bad_vertex"] <= case.hub


def test_parents(case):
    for src in case.srcs.tolist():
        par = O.bfs_det_parent(case.off, case.edg, src, "min")
        d = torch.from_numpy(par.view(np.int32)).cuda()
        assert case.dg.check(src, d)["bad_vertex"] == pb.NONE
        v = case.hub if src != case.hub else int(case.edg[-1])  # an end of the last list
        bad = par.copy()
        bad[v] = pb.NONE
        want = O.check_bfs(case.off, case.edg, src, bad)
        assert want >= 0
        assert case.dg.check(src, torch.from_numpy(bad.view(np.int32)).cuda())["bad_vertex"] == want


@pytest.mark.parametrize("direction,chunk", [(pb.DIR_AUTO, 8), (pb.DIR_TOPDOWN, 8), (pb.DIR_TOPDOWN, 32),
                                             (pb.DIR_TOPDOWN, 1 << 20), (pb.DIR_BOTTOMUP, 32)])
def test_search(searched, direction, chunk):
    """Both ways to expand a list and the probes from the other side; a chunk degree past every list's length is
    lowered so near the limit."""
    c = searched
    for src in c.srcs[:2].tolist():
        want = O.bfs_levels(c.off, c.edg, src)
        for mode, rule in ((pb.PARENT_ANY, None), (pb.PARENT_MIN, "min"), (pb.PARENT_MAX, "max")):
            par, lv, st = c.dg.bfs(src, parent_mode=mode, direction=direction, levels=True, chunk_min_degree=chunk)
            assert np.array_equal(lv, want)
            if rule:
                assert np.array_equal(par.view(np.uint32), O.bfs_det_parent(c.off, c.edg, src, rule))
            else:
                assert O.check_bfs(c.off, c.edg, src, par.view(np.uint32)) == -1
            assert st["visited"] == int((want != pb.NONE).sum())


@pytest.mark.parametrize("k", [4, 100, 200])
@pytest.mark.parametrize("direction", [pb.DIR_AUTO, pb.DIR_TOPDOWN, pb.DIR_BOTTOMUP])
def test_batch(searched, k, direction):
    """One, two and four mask words, by pushes and by pulls."""
    c = searched
    srcs = np.concatenate([c.srcs, np.arange(PAIRED, PAIRED + k - 4)]).astype(np.uint32)
    rows, _ = c.dg.bfs_multi(srcs, direction=direction)
    assert np.array_equal(rows, O.levels_u8(c.off, c.edg, srcs))


def test_searches_refuse_more_edges(case):
    with pytest.raises(pb.PbgError, match="PBG_MAX_SEARCH_EDGES"):
        case.dg.bfs(case.hub)
    with pytest.raises(pb.PbgError, match="PBG_MAX_SEARCH_EDGES"):
        case.dg.bfs_multi(case.srcs)
