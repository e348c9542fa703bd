"""The rules of a context's device scratch (gsofa_scratch.hpp), on a fake
device; and on a GPU, jobs whose budget ends just where their optional scratch
does."""
import functools
import os
import subprocess
import time

import numpy as np
import pytest

import gsofa_b200
import oracle
from gsofa_b200 import matgen
from gsofa_b200.matgen import Graph
from tests.common import assert_same

HERE = os.path.dirname(os.path.abspath(__file__))


def test_nothing_that_a_job_has_taken_is_freed(tmp_path):
    exe = str(tmp_path / "scratch_rules")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", exe, os.path.join(HERE, "scratch_rules.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def _snapshots_used(g, budget):
    """Whether a counts-only job under this budget keeps snapshots."""
    with gsofa_b200.Context(0, mem_budget_bytes=budget) as ctx:
        r = ctx.symbfact(ctx.upload(g), want_pattern=0)
        return r.cycles[2] > 0


@pytest.mark.gpu
def test_jobs_whose_budget_ends_just_where_their_snapshots_do():
    g = matgen.grid3d(32, 24, 16, seed=6)      # 12,288 lines: snapshots are a twentieth of the scratch
    ref = oracle.symbfact(g.beg, g.end, g.adj, want_pattern=False)
    tiny = [matgen.grid2d(3, seed=i) for i in range(40)]
    tiny_refs = [oracle.symbfact(t.beg, t.end, t.adj, want_pattern=False) for t in tiny]
    lo, hi = 10 << 20, 64 << 20
    assert _snapshots_used(g, hi) and not _snapshots_used(g, lo)
    while hi - lo > 64:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _snapshots_used(g, mid) else (mid, hi)
    for budget in [hi + d for d in range(-2048, 4096, 256)] + [hi + (1 << k) for k in range(13, 18)]:
        with gsofa_b200.Context(0, mem_budget_bytes=budget) as ctx:
            m = ctx.upload(g)
            for _ in range(2):
                r = ctx.symbfact(m, want_pattern=0)
                assert r.fill_count == ref["fill_count"], budget
                assert np.array_equal(r.u_row_count, ref["u_row_count"]), budget
                assert np.array_equal(r.l_col_count, ref["l_col_count"]), budget
            # a larger job, which needs more for its descriptors, where the
            # first one's snapshots are still held
            rs = ctx.symbfact_batch([m] + [ctx.upload(t) for t in tiny], want_pattern=0)
            for r, want in zip(rs, [ref] + tiny_refs):
                assert r.fill_count == want["fill_count"], budget
                assert np.array_equal(r.l_col_count, want["l_col_count"]), budget


@pytest.mark.gpu
def test_a_pattern_that_fits_nowhere_is_refused_after_one_run():
    """The lists of the 48^3 stencil take 708 MB with their compacted copy; a
    context with less runs the job once to learn that, not once for every
    number of CTAs."""
    g = matgen.grid3d(48, seed=3)
    with gsofa_b200.Context(0, mem_budget_bytes=600 << 20) as ctx:
        m = ctx.upload(g)
        took = []
        for _ in range(3):
            t = time.perf_counter()
            with pytest.raises(gsofa_b200.GsofaError) as e:
                ctx.symbfact(m)
            took.append(time.perf_counter() - t)
            assert e.value.status == 2
        # a run at full width takes 1.3 ms; all numbers of CTAs some 700
        assert min(took) < 0.1, took
        # counts need no pool; and once they are known, nothing runs in vain
        assert ctx.symbfact(m, want_pattern=0).nnz_lu > 88_000_000
        with pytest.raises(gsofa_b200.GsofaError):
            ctx.symbfact(m)


@pytest.mark.gpu
@pytest.mark.parametrize("mib", [200, 260, 320, 400, 600])
def test_a_pattern_that_fits_beside_fewer_ctas(mib):
    """Where lists and traversals do not fit together at full width, the job is
    run on the CTAs that do, on a context that has met the matrix or not."""
    g = matgen.grid3d(32, seed=4)              # 32,768 lines; lists 19.6M entries, 157 MB with their copy
    ref = oracle.symbfact(g.beg, g.end, g.adj)
    with gsofa_b200.Context(0, mem_budget_bytes=mib << 20) as ctx:
        m = ctx.upload(g)
        for _ in range(2):
            assert_same(ctx.symbfact(m), ref, where=f"{mib} MiB")
        assert_same(ctx.symbfact(ctx.upload(g)), ref, where=f"{mib} MiB, once more")
        small = matgen.grid2d(20, seed=1)
        assert_same(ctx.symbfact(ctx.upload(small)), oracle.symbfact(small.beg, small.end, small.adj), where="small")
        assert_same(ctx.symbfact(m), ref, where=f"{mib} MiB, after a small one")


def _least_budget(g, **kw):
    """The smallest budget, to a KiB, under which the job runs."""
    lo, hi = 1 << 20, 1 << 30
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        with gsofa_b200.Context(0, mem_budget_bytes=mid) as ctx:
            try:
                ctx.symbfact(ctx.upload(g), **kw)
                hi = mid
            except gsofa_b200.GsofaError as e:
                assert e.status == 2
                lo = mid
    return hi


@pytest.mark.gpu
def test_lists_need_a_row_of_stamps_and_no_more():
    """Beside what counts take, the least that a job with lists runs in is its
    pool and one row of stamps for each of two traversals."""
    n = 100_000
    end = np.concatenate([np.arange(2, 2 * n, 2), [2 * n - 2]]).astype(np.int32)
    end[0] = 1
    end[1:-1] = np.arange(3, 2 * n - 2, 2)
    beg = np.concatenate([[0], end[:-1]]).astype(np.int32)
    adj = np.concatenate([[1], np.stack([np.arange(n - 2), np.arange(2, n)], 1).ravel(), [n - 2]]).astype(np.int32)
    g = Graph(n, beg, end, adj, "path")
    row = 2 * ((n + 4095) // 4096 * 4096)
    assert _least_budget(g) - _least_budget(g, want_pattern=0) <= 2 * row + (8 << 20) + 4096


@pytest.mark.gpu
@pytest.mark.parametrize("make", [functools.partial(matgen.grid2d, 37, drop_frac=0.1, seed=5),
                                  functools.partial(matgen.grid3d, 23, 21, 19, seed=6),
                                  functools.partial(matgen.powerlaw, 3001, seed=4),
                                  functools.partial(matgen.bordered_blocks, 100, seed=2)],
                         ids=["grid2d", "nd3d", "powerlaw", "bordered"])
@pytest.mark.parametrize("flags", [0, gsofa_b200.FLAG_GLOBAL_STATE], ids=["shared", "global"])
def test_lists_at_every_budget(make, flags):
    """From the least budget on: one row of stamps a traversal, then two, and
    few CTAs to all."""
    g = make()
    ref = oracle.symbfact(g.beg, g.end, g.adj)
    ctas = set()
    budget = _least_budget(g, flags=flags)
    while budget < 256 << 20:
        for reuse in (-1, 2):
            with gsofa_b200.Context(0, mem_budget_bytes=budget) as ctx:
                m = ctx.upload(g)
                for _ in range(2):
                    r = ctx.symbfact(m, flags=flags, reuse=reuse)
                    assert_same(r, ref, where=f"{g.name} budget {budget} reuse {reuse}")
            ctas.add(r.ctas)
        budget += budget // 12
    assert len(ctas) > 4


@pytest.mark.gpu
def test_what_a_job_left_gives_way_to_other_calls():
    """A job takes all the CTAs that a small budget holds; an ordering, a larger
    upload and the streamed form find room on the same context all the same."""
    import torch
    g = matgen.grid3d(21, seed=3)
    ref = oracle.symbfact(g.beg, g.end, g.adj)
    # the ordering takes about 5 MiB (two arrays of 141,000 keys, columns, sort
    # space); the job's traversals fill what its lists (19 MiB with their copy) leave
    big = matgen.powerlaw(8000, seed=1, ordering="random")
    with gsofa_b200.Context(0) as ctx:
        perm = ctx.order_rcm(big)
    for mib in (32, 36, 44):
        with gsofa_b200.Context(0, mem_budget_bytes=mib << 20) as ctx:
            m = ctx.upload(g)
            assert_same(ctx.symbfact(m), ref, where=f"{mib} MiB")
            assert np.array_equal(ctx.order_rcm(big), perm)
            assert_same(ctx.symbfact(m), ref, where=f"{mib} MiB, after an ordering")
            ctx.upload(big).free()
            pool = torch.zeros(ref["u_idx"].size + ref["l_idx"].size, dtype=torch.int32).pin_memory().numpy()
            for _ in range(2):
                r = ctx.symbfact_ranges(m, pool)
                assert np.array_equal(r.u_row_count, ref["u_row_count"])
                for v in (0, 100, 5000, 9000):
                    assert np.array_equal(r.u_row(v), ref["u_idx"][ref["u_ptr"][v]:ref["u_ptr"][v + 1]])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8000, 50_000, 200_000, 800_000, 1_000_000])
def test_predicted_scratch_covers_a_job_with_lists(n):
    import torch
    v = np.arange(n, dtype=np.int32)
    g = Graph(n, v, v + 1, (v ^ 1).astype(np.int32), "pairs")
    pool = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    with gsofa_b200.Context(0) as ctx:
        m = ctx.upload(g)
        predicted = ctx.predict_scratch_bytes(n, g.nnz)
        free = torch.cuda.mem_get_info()[0]
        ctx.symbfact_ranges(m, pool)
        used = free - torch.cuda.mem_get_info()[0]
    # beside it: snapshots, one byte in thirteen, and the 2 MiB that each of a
    # dozen allocations is rounded to
    assert used <= predicted * 13 / 12 + (28 << 20)
    assert predicted <= used * 2 + (28 << 20)
