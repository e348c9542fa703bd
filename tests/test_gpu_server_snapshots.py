"""When the serving kernel's snapshots give way to a request's memory."""
import numpy as np
import pytest

import gsofa_b200
import oracle
from gsofa_b200 import matgen
from gsofa_b200.matgen import Graph

pytestmark = pytest.mark.gpu

BASE = matgen.grid2d(25, seed=1)


def _of_size(nnz):
    """The grid with its first line's first id repeated up to nnz entries."""
    more = nnz - BASE.nnz
    adj = np.concatenate([np.full(more, BASE.adj[BASE.beg[0]], np.int32)] +
                         [BASE.adj[b:e] for b, e in zip(BASE.beg, BASE.end)])
    lens = (BASE.end - BASE.beg).astype(np.int64)
    lens[0] += more
    end = np.cumsum(lens).astype(np.int32)
    return Graph(BASE.n, (end - lens).astype(np.int32), end, adj.astype(np.int32), "sized")


def _server():
    return gsofa_b200.StreamServer(0, mem_budget_bytes=256 << 20, max_n=1000)


def _done(srv, rid):
    while rid not in srv.poll():
        pass


def _held_at_once(srv, g):
    """How many such requests the server takes before the first one is polled
    for: while it may be running, the snapshots stay."""
    ids = []
    while (rid := srv.submit(g)) is not None:
        ids.append(rid)
    return ids


def test_a_request_that_never_fits_leaves_the_snapshots_in_place():
    # the arena is some 45 MB, the snapshots 3.6 MB, a request of 40,000
    # entries half a MB, one of 12,000,000 entries 100 MB and more
    g = _of_size(40_000)
    ref = oracle.symbfact(BASE.beg, BASE.end, BASE.adj, want_pattern=False)
    with _server() as srv:
        room = len(_held_at_once(srv, g))
    with _server() as srv:
        assert srv.submit(_of_size(12_000_000)) is None
        ids = _held_at_once(srv, g)
        assert len(ids) == room
        left = set(ids)
        while left:
            left -= set(srv.poll())
        for rid in ids[1:]:
            r = srv.result(rid)
            assert r.fill_count == ref["fill_count"] and np.array_equal(r.u_row_count, ref["u_row_count"])


def test_a_result_that_waits_to_be_fetched_does_not_keep_the_snapshots():
    small = _of_size(4_000)
    with _server() as srv:
        lo, hi = 40_000, 12_000_000          # entries that fit an empty server, and that don't
        while hi - lo > 4_000:
            mid = (lo + hi) // 2
            rid = srv.submit(_of_size(mid))
            if rid is None:
                hi = mid
            else:
                lo = mid
                _done(srv, rid)
                srv.result(rid)
    with _server() as srv:
        first = srv.submit(small)
        _done(srv, first)
        big = _of_size(lo - 3 * (srv.request_bytes(small.n, small.nnz) // 4))
        rid = srv.submit(big)
        assert rid is not None
        _done(srv, rid)
        a, b = srv.result(first), srv.result(rid)
        assert a.fill_count == b.fill_count and np.array_equal(a.l_col_count, b.l_col_count)
