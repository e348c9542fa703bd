"""The traversal kernel's own edges, against the oracle: runs of consecutive
sources (windows of 31), units and pieces of sources shared between CTAs, row
slots and long rows, chains of lists around a batch of 32, snapshots, and the
same with bitmaps in global memory, wide blocks, fixed pieces and a budget too
small for the optional scratch."""
import functools

import numpy as np
import pytest

import gsofa_b200
import oracle
from gsofa_b200 import matgen
from gsofa_b200.matgen import Graph
from tests.common import assert_same, random_graph

pytestmark = pytest.mark.gpu


def _rows(n, rows, name):
    """A symmetric pattern from its upper rows (row v: ids above v)."""
    full = [set() for _ in range(n)]
    for v, r in enumerate(rows):
        for u in r:
            full[v].add(u)
            full[u].add(v)
    lens = np.array([len(r) for r in full], np.int32)
    end = np.cumsum(lens, dtype=np.int64).astype(np.int32)
    adj = np.array([u for r in full for u in sorted(r)], np.int32)
    return Graph(n, end - lens, end, adj, name)


def path(n):
    return _rows(n, [[v + 1] if v + 1 < n else [] for v in range(n)], f"path_{n}")


def wide_rows(n, width):
    """Every `width`-th line meets the next `width` lines: rows longer than a
    warp's queue share, and chains that hold for one block each."""
    return _rows(n, [list(range(v + 1, min(n, v + width + 1))) if v % width == 0 else [min(v + 1, n - 1)] * (v + 1 < n)
                     for v in range(n)], f"wide_{n}_{width}")


CASES = ([functools.partial(path, n) for n in (1, 2, 8, 31, 32, 33, 34, 63, 64, 65, 255, 256, 257, 9001)] +
         [functools.partial(wide_rows, 1500, w) for w in (31, 32, 33, 513)] +
         [functools.partial(matgen.grid2d, 37, drop_frac=0.1, seed=5),
          functools.partial(matgen.grid3d, 23, 21, 19, seed=6),         # snapshots: separators leave and return
          functools.partial(random_graph, 260, 0.015, 11),              # free-form layout, mean degree about 4
          functools.partial(random_graph, 9001, 0.0002, 12),            # low degree, past 8K lines
          functools.partial(matgen.powerlaw, 8193, seed=4)])


@pytest.mark.parametrize("case", range(len(CASES)))
def test_traversals_match_oracle(case):
    g = CASES[case]()
    ref = oracle.symbfact(g.beg, g.end, g.adj)
    with gsofa_b200.Context(0) as ctx:
        m = ctx.upload(g)
        for kw in ({}, {"flags": gsofa_b200.FLAG_GLOBAL_STATE}, {"flags": gsofa_b200.FLAG_WIDE_REGS},
                   {"block_size": 256}, {"src_chunk": 37}, {"reuse": 2}, {"reuse": 0}):
            if kw.get("block_size") == 256 and g.n > 8192:
                continue
            where = f"{g.name} {kw}"
            assert_same(ctx.symbfact(m, **kw), ref, where=where)
            r = ctx.symbfact(m, want_pattern=0, **kw)
            assert r.fill_count == ref["fill_count"] and r.n_supernodes == ref["sn_start"].size, where
            assert np.array_equal(r.u_row_count, ref["u_row_count"]), where
            assert np.array_equal(r.l_col_count, ref["l_col_count"]), where
            assert np.array_equal(r.line_flags, ctx.symbfact(m, want_pattern=0, reuse=0).line_flags), where


def test_shared_pieces_of_a_batch_and_of_a_line_range():
    """Pieces of several matrices in one launch, and of a range of lines whose
    ends are no multiple of a unit."""
    gs = [path(9001), matgen.grid3d(21, seed=3), matgen.powerlaw(3001, seed=7), path(1), matgen.grid2d(97, seed=2)]
    refs = [oracle.symbfact(g.beg, g.end, g.adj, want_pattern=False) for g in gs]
    with gsofa_b200.Context(0) as ctx:
        ms = [ctx.upload(g) for g in gs]
        for r, ref, g in zip(ctx.symbfact_batch(ms, want_pattern=0), refs, gs):
            assert r.fill_count == ref["fill_count"], g.name
            assert np.array_equal(r.u_row_count, ref["u_row_count"]), g.name
            assert np.array_equal(r.l_col_count, ref["l_col_count"]), g.name
        for lo, hi in ((3, 9000), (4095, 4097), (8999, 9261)):
            r = ctx.symbfact(ms[1], want_pattern=0, line_lo=lo, line_hi=hi)
            assert np.array_equal(r.u_row_count[lo:hi], refs[1]["u_row_count"][lo:hi]), (lo, hi)
            assert np.array_equal(r.l_col_count[lo:hi], refs[1]["l_col_count"][lo:hi]), (lo, hi)


def test_a_small_budget_gives_up_the_optional_scratch_only():
    g = matgen.grid3d(21, seed=3)
    ref = oracle.symbfact(g.beg, g.end, g.adj)
    for mib in (24, 40, 48, 96, 512):
        with gsofa_b200.Context(0, mem_budget_bytes=mib << 20) as ctx:
            assert_same(ctx.symbfact(ctx.upload(g)), ref, where=f"{mib} MiB")


def test_the_server_gives_its_snapshots_up_for_a_request_that_needs_their_room():
    """Requests grow (by repeated entries) in steps below the snapshots' size
    until the server has no room: one of them takes the snapshots' place."""
    base = matgen.grid2d(25, seed=1)
    ref = oracle.symbfact(base.beg, base.end, base.adj, want_pattern=False)
    rows = [base.adj[b:e] for b, e in zip(base.beg, base.end)]
    grown = 0
    with gsofa_b200.StreamServer(0, mem_budget_bytes=256 << 20, max_n=1000) as srv:
        for k in range(200, 6000, 40):
            adj = np.concatenate([np.tile(r, 3 * k) if v % 3 == 0 else r for v, r in enumerate(rows)])
            lens = np.array([len(r) * (3 * k if v % 3 == 0 else 1) for v, r in enumerate(rows)], np.int64)
            end = np.cumsum(lens).astype(np.int32)
            rid = srv.submit(Graph(base.n, (end - lens).astype(np.int32), end, adj.astype(np.int32), "grown"))
            if rid is None:
                break
            while rid not in srv.poll():
                pass
            r = srv.result(rid)
            assert r.fill_count == ref["fill_count"] and np.array_equal(r.u_row_count, ref["u_row_count"]), k
            grown += 1
        else:
            pytest.fail("the server never ran out of room")
    assert grown > 0
