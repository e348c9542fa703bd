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


def _inspected(n, rows, lengths):
    """Input entries of every source's line and of the lines that its traversal expands."""
    total = 0
    for s in range(n):
        seen, todo = {s}, [s]
        while todo:
            v = todo.pop()
            total += lengths[v]
            for u in rows[v]:
                if u < s and u not in seen:
                    seen.add(u)
                    todo.append(u)
    return total


@pytest.mark.parametrize("flags", [0, gsofa_b200.FLAG_GLOBAL_STATE], ids=["shared", "global"])
@pytest.mark.parametrize("level", [1, 21], ids=["leader", "helpers"])
@pytest.mark.parametrize("longer", [0, 30], ids=["slot", "long_row"])
def test_work_that_one_lane_counts_past_2_32(flags, level, longer):
    """Line 0 repeats one id 2^25 times, and every other line's traversal
    expands it: 260 of them in a piece are 8.7e9 input entries, all in the same
    lane's count.  With `longer` line 0's row does not fit a slot; with a first
    level of 21 vertices it is the helper warps that expand it."""
    n, copies = 260, 1 << 25
    rows = [sorted(set(range(1, longer + 1)) | {n - 1})] + [list(range(min(v, level))) for v in range(1, n)]
    lengths = [longer + copies] + [len(r) for r in rows[1:]]
    adj = [np.arange(1, longer + 1, dtype=np.int32), np.full(copies, n - 1, np.int32)]
    adj += [np.array(r, np.int32) for r in rows[1:]]
    end = np.cumsum(lengths, dtype=np.int64).astype(np.int32)
    beg = np.concatenate([[0], end[:-1]]).astype(np.int32)
    with gsofa_b200.Context(0) as ctx:
        m = ctx.upload(Graph(n, beg, end, np.concatenate(adj), "copies"))
        r = ctx.symbfact(m, want_pattern=0, reuse=0, src_chunk=512, flags=flags)
        assert r.e_insp == _inspected(n, rows, lengths)
        assert r.e_insp > 1 << 32
