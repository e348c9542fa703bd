"""The largest matrices whose visited bitmaps fit in shared memory, two of them
(839,680 lines) or one (1,736,704), under the options that ask for it."""
import numpy as np
import pytest

import gsofa_b200
import oracle
from gsofa_b200.matgen import Graph
from tests.common import assert_same

pytestmark = pytest.mark.gpu

PAIR, SINGLE = 839_680, 1_736_704      # bitmaps are multiples of 4096 lines
SHARED, WIDE = gsofa_b200.FLAG_SHARED_STATE, gsofa_b200.FLAG_WIDE_REGS


def _paths_and_hub(n, block=64, spokes=3000):
    """Paths of 64 lines, and a last line that meets one line of each of the
    first 3,000: its traversal's levels pass the frontier's shared memory."""
    v = np.arange(n - 2, dtype=np.int64)
    v = v[v % block != block - 1]
    hub = np.arange(spokes, dtype=np.int64) * block + 17
    u = np.concatenate([v, v + 1, hub, np.full(spokes, n - 1)])
    w = np.concatenate([v + 1, v, np.full(spokes, n - 1), hub])
    order = np.lexsort((w, u))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(u, minlength=n), out=ptr[1:])
    return Graph.from_csr(ptr, w[order].astype(np.int32), f"paths_{n}")


@pytest.fixture(scope="module", params=[PAIR, SINGLE])
def case(request):
    g = _paths_and_hub(request.param)
    return g, oracle.symbfact(g.beg, g.end, g.adj)


def test_sizes_that_fit_are_taken(case):
    g, ref = case
    blocks = [{"block_size": b, "flags": SHARED} for b in (256, 512, 768, 1024)]
    if g.n == PAIR:
        options = [{"flags": SHARED}, {"flags": WIDE}, {"flags": WIDE | SHARED}, {"block_size": 768},
                   {"block_size": 1024}] + blocks
    else:
        options = [{"flags": SHARED}, {"flags": SHARED, "reuse": 2}, {"reuse": 2, "block_size": 768},
                   {"reuse": 2, "block_size": 1024}, {"reuse": 2}] + blocks
    with gsofa_b200.Context(0) as ctx:
        m = ctx.upload(g)
        for kw in options:
            r = ctx.symbfact(m, **kw)
            assert_same(r, ref, where=f"{g.n} {kw}")
            assert r.ctas == 148, kw                 # the bitmaps fill an SM
            c = ctx.symbfact(m, want_pattern=0, **kw)
            assert np.array_equal(c.u_row_count, ref["u_row_count"]), kw
            assert np.array_equal(c.l_col_count, ref["l_col_count"]), kw


def test_the_server_in_shared_memory_takes_what_it_took():
    with gsofa_b200.StreamServer(0, flags=SHARED, max_n=794_624) as srv:
        assert srv.max_n == 794_624
        g = _paths_and_hub(794_624)
        ref = oracle.symbfact(g.beg, g.end, g.adj, want_pattern=False)
        rid = srv.submit(g)
        while rid not in srv.poll():
            pass
        r = srv.result(rid)
        assert r.fill_count == ref["fill_count"] and np.array_equal(r.l_col_count, ref["l_col_count"])
    with gsofa_b200.StreamServer(0, flags=SHARED) as srv:
        assert srv.max_n >= 794_624
