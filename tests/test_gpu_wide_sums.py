"""Sums that pass 32 bits: the entries of a chain's lists, and the work that one
lane of a warp counts in a piece."""
import numpy as np
import pytest
import torch

import gsofa_b200
from gsofa_b200.matgen import Graph

pytestmark = pytest.mark.gpu


@pytest.mark.slow
def test_a_chain_of_lists_with_more_than_2_32_entries():
    """Line 0 meets every line and line v meets v - 1, so every U row is full;
    64 lists of one chain, which go out together, hold 4.3e9 entries."""
    n, lo, hi = 67_200_000, 64, 160
    beg = np.empty(n, np.int32)
    beg[0] = 0
    beg[1:] = np.arange(n - 1, 2 * n - 2, dtype=np.int32)
    end = np.empty(n, np.int32)
    end[:-1] = beg[1:]
    end[-1] = 2 * n - 2
    adj = np.empty(2 * n - 2, np.int32)
    adj[:n - 1] = np.arange(1, n, dtype=np.int32)
    adj[n - 1:] = np.arange(n - 1, dtype=np.int32)
    entries = (hi - lo) * (n - hi) + (hi - lo) * (hi - lo - 1) // 2 + (hi - lo)
    pool = torch.full((entries + 1024,), -1, dtype=torch.int32, device="cuda")
    line = torch.arange(n, dtype=torch.int32, device="cuda")
    with gsofa_b200.Context(0, mem_budget_bytes=30 << 30) as ctx:
        m = ctx.upload(Graph(n, beg, end, adj, "full"))
        r = ctx.symbfact_ranges(m, pool, line_lo=lo, line_hi=hi, src_chunk=128)
        assert r.pool_used == entries
        for s in range(lo, hi):
            u, c = int(r.u_beg[s]), int(r.u_row_count[s])
            assert c == n - 1 - s and torch.equal(pool[u:u + c], line[s + 1:]), s
            assert r.l_col_count[s] == 1 and int(pool[int(r.l_beg[s])]) == s + 1, s
    assert bool((pool[entries:] == -1).all())
