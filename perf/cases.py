"""What this library is used for, as cases that can be timed.

Each case is one call (or one short sequence of calls) that a program using
``gsofa_b200`` makes, on seeded synthetic matrices of the kinds the library's
benchmarks and tests use: 5-point grids in natural order, 7-point grids in
nested-dissection order, circuit-like power-law patterns in reverse
Cuthill-McKee order, bordered block-diagonal patterns, and mixes of them.
``listed()`` names the cases, ``draw()`` gives others of the same ranges.
Buffers a program keeps are sized by the case, not by one seed's result, and
come back whole (zeros behind what was written).

Every output is a whole number: counts, indices, flags.  There is nothing to
round, so there is no ``exact()``.
"""
import functools
import math

import numpy as np
import torch

import gsofa_b200
from gsofa_b200 import matgen

DROP = 0.1          # share of off-diagonal pairs that lose one side


def listed():
    return [
        # Code inside another framework that owns the device memory factorizes
        # one small subproblem whose arrays are on the device already: the
        # smallest call, all latency.
        dict(name="noalloc_grid2d_33x31", call="noalloc", kind="grid2d", nx=33, ny=31),
        # A small matrix with the whole pattern fetched into the caller's
        # page-locked buffers as row and column lists: the 64 x 64 grid.
        dict(name="csr_grid2d_64x64", call="csr", kind="grid2d", nx=64, ny=64),
        # Sizing a solver's factors: counts and supernodes of an ordinary 3-D
        # problem with ragged sides.
        dict(name="counts_nd3d_31x29x27", call="counts", kind="nd3d", nx=31, ny=29, nz=27),
        # The same at the benchmark's size.
        dict(name="counts_nd3d_80x80x80", call="counts", kind="nd3d", nx=80, ny=80, nz=80),
        # The benchmark's own call: the whole pattern of the 80^3 problem into
        # a device pool, then put in line order there, as a numeric phase on
        # the device that walks the lines needs it.
        dict(name="ranges_nd3d_80x80x80", call="ranges", kind="nd3d", nx=80, ny=80, nz=80),
        # A solver that meets each matrix once: upload from page-locked host
        # memory, factorize, fetch the supernodal structure, free.
        dict(name="solve_nd3d_47x48x49", call="supernodal", kind="nd3d", nx=47, ny=48, nz=49),
        # Circuit simulation: counts of a large power-law pattern, whose fill
        # is a quarter of a dense matrix (large frontiers, long lists).
        dict(name="counts_powerlaw_200003", call="counts", kind="powerlaw", n=200003),
        # ... and the whole pattern of a smaller one.
        dict(name="ranges_powerlaw_20011", call="ranges", kind="powerlaw", n=20011),
        # Many mid-size matrices of mixed kinds in one launch, replayed from a
        # CUDA graph while the batch stays the same.
        dict(name="batch_20_mixed", call="batch", kind="mix", count=20, n_lo=2000, n_hi=50000, mix=4),
        # A burst of small requests through the persistent serving kernel.
        dict(name="serve_32_mixed", call="serve", kind="mix", count=32, n_lo=1000, n_hi=20000, mix=5),
        # More lines than two visited bitmaps in shared memory hold.
        dict(name="counts_bordered_864008", call="counts", kind="bordered", blocks=27000),
        # The ordering step before the factorization.
        dict(name="order_powerlaw_120011", call="order", kind="powerlaw", n=120011),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["noalloc", "csr", "counts", "counts", "counts", "ranges", "ranges", "supernodal", "batch",
                       "serve", "order"])
    if call == "noalloc":
        nx = _log_uniform(rng, 8, 110)
        return dict(call=call, kind="grid2d", nx=nx, ny=max(4, nx - rng.randint(0, nx // 3)))
    if call == "order":
        return dict(call=call, kind="powerlaw", n=_log_uniform(rng, 2000, 150000))
    if call == "batch":
        return dict(call=call, kind="mix", count=rng.randint(4, 24), n_lo=2000, n_hi=_log_uniform(rng, 5000, 50000),
                    mix=rng.randrange(1 << 20))
    if call == "serve":
        return dict(call=call, kind="mix", count=rng.randint(4, 40), n_lo=1000, n_hi=_log_uniform(rng, 2000, 20000),
                    mix=rng.randrange(1 << 20))
    if call == "csr":
        nx = _log_uniform(rng, 12, 130)
        return dict(call=call, kind="grid2d", nx=nx, ny=max(4, nx - rng.randint(0, nx // 3)))
    kind = rng.choice(["grid2d", "nd3d", "nd3d", "powerlaw", "powerlaw", "bordered"])
    if call == "supernodal" and kind in ("bordered", "grid2d"):
        kind = "nd3d"
    if kind == "grid2d":
        nx = _log_uniform(rng, 40, 400 if call == "counts" else 200)
        return dict(call=call, kind=kind, nx=nx, ny=max(4, nx - rng.randint(0, nx // 3)))
    if kind == "nd3d":
        a = _log_uniform(rng, 8, 80 if call != "supernodal" else 50)
        b, c = (max(4, a - rng.randint(0, a // 4)) for _ in range(2))
        return dict(call=call, kind=kind, nx=a, ny=b, nz=c)
    if kind == "powerlaw":
        return dict(call=call, kind=kind, n=_log_uniform(rng, 1500, 180000 if call == "counts" else 20000))
    return dict(call=call, kind=kind, blocks=_log_uniform(rng, 300, 30000))


# ----------------------------------------------------------------------------
# Inputs


@functools.lru_cache(maxsize=4)
def _grid(dims, nested):
    """The grid's off-diagonal entries in line order: rows, columns, and the
    undirected pair each entry belongs to (2 * pair + side)."""
    n, u, v = matgen._grid_edges(dims)
    if nested:
        new = matgen.nested_dissection_order(dims)
        u, v = new[u], new[v]
    pair = np.arange(u.shape[0], dtype=np.int64)
    rows, cols = np.concatenate([u, v]), np.concatenate([v, u])
    tag = np.concatenate([2 * pair, 2 * pair + 1])
    diag = np.arange(n, dtype=np.int64)
    rows, cols = np.concatenate([rows, diag]), np.concatenate([cols, diag])
    tag = np.concatenate([tag, np.full(n, -1, np.int64)])
    order = np.argsort(rows * n + cols, kind="stable")
    return n, u.shape[0], rows[order], cols[order].astype(np.int32), tag[order]


def _grid_graph(dims, nested, seed):
    n, pairs, rows, cols, tag = _grid(dims, nested)
    rng = np.random.default_rng(seed)
    lost = np.where(rng.random(pairs) < DROP, rng.integers(0, 2, pairs), -1)   # the side a pair loses
    keep = (tag < 0) | (lost[tag >> 1] != (tag & 1))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows[keep], minlength=n), out=ptr[1:])
    return matgen.Graph.from_csr(ptr, cols[keep], "grid")


def _graph(case, seed):
    kind = case["kind"]
    if kind == "grid2d":
        return _grid_graph((case["nx"], case["ny"]), False, seed)
    if kind == "nd3d":
        return _grid_graph((case["nx"], case["ny"], case["nz"]), True, seed)
    if kind == "powerlaw":
        return matgen.powerlaw(case["n"], seed=seed, ordering="random" if case["call"] == "order" else "rcm")
    return matgen.bordered_blocks(case["blocks"], seed=seed)


def _mix(case, seed):
    """The mix's kinds and sizes are the case's (`mix`), its patterns the seed's."""
    spec = matgen.mixed_spec(case["count"], case["n_lo"], case["n_hi"], case["mix"])
    return [matgen.make(kind, n, seed + i) for i, (kind, n, _) in enumerate(spec)]


def _capacity(case):
    """Pattern entries that a pool for this case has room for."""
    n, _, entries = _shape(case)
    return int((1.4 if case["kind"] == "powerlaw" else 1.1) * entries) + 64 * n


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _pinned_empty(count, dtype):
    return torch.zeros(max(int(count), 1), dtype=dtype).pin_memory().numpy()


def prepare(case, seed):
    s = dict(call=case["call"])
    if case["call"] == "serve":
        s["graphs"] = _mix(case, seed)
        s["server"] = gsofa_b200.StreamServer(0, mem_budget_bytes=4 << 30, max_n=65536)
        return s
    if case["call"] == "batch":
        ctx = s["ctx"] = gsofa_b200.Context(0)
        s["mats"] = [ctx.upload(g) for g in _mix(case, seed)]
        s["params"] = gsofa_b200.Params.default(want_pattern=0, flags=gsofa_b200.FLAG_GRAPH)
        return s
    g = _graph(case, seed)
    if case["call"] == "noalloc":
        dev = torch.device("cuda", 0)
        s["n"], s["nnz"] = g.n, g.nnz
        s["in"] = [torch.from_numpy(a).to(dev) for a in (g.beg, g.end, g.adj)]
        s["out"] = [torch.zeros(g.n, dtype=torch.int32, device=dev) for _ in range(3)]
        return s
    ctx = s["ctx"] = gsofa_b200.Context(0)
    if case["call"] == "order":
        s["graph"] = g
        return s
    if case["call"] == "supernodal":
        s["graph"] = matgen.Graph(g.n, _pinned(g.beg), _pinned(g.end), _pinned(g.adj), g.name)
        room = dict(xsup=g.n + 1, supno=g.n, xlsub=g.n + 1, lsub=_capacity(case) // 2, xusub=g.n + 1,
                    usub=_capacity(case) // 2)
        s["buffers"] = {k: _pinned_empty(c, torch.int64 if k in ("xlsub", "xusub") else torch.int32)
                        for k, c in room.items()}
        return s
    s["matrix"] = ctx.upload(g)
    if case["call"] == "csr":
        half = _capacity(case) // 2
        room = dict(u_row_count=g.n, l_col_count=g.n, l_row_count=g.n, sn_start=g.n, u_idx=half, l_idx=half)
        s["buffers"] = {k: _pinned_empty(c, torch.int32) for k, c in room.items()}
        s["buffers"].update({k: _pinned_empty(g.n + 1, torch.int64) for k in ("u_ptr", "l_ptr")})
        s["params"] = gsofa_b200.Params.default()
    if case["call"] == "ranges":
        s["stream"] = torch.cuda.Stream()   # the program's own work and the library's in one order
        ctx.set_stream(s["stream"].cuda_stream)
        s["pool"] = torch.empty(_capacity(case), dtype=torch.int32, device="cuda")
        s["place"] = torch.arange(_capacity(case), dtype=torch.int32, device="cuda")
        s["lines"] = torch.zeros_like(s["pool"])
        s["buffers"] = {k: _pinned_empty(g.n, torch.int32)
                        for k in ("u_row_count", "l_col_count", "l_row_count", "sn_start")}
        s["buffers"].update({k: _pinned_empty(g.n, torch.int64) for k in ("u_beg", "l_beg")})
        s["params"] = gsofa_b200.Params.default()
    return s


# ----------------------------------------------------------------------------
# One pass


def _lines(r):
    """A counts-only result: totals, counts and link flags of every line, supernodes."""
    return dict(fill_count=r.fill_count, nnz_lu=r.nnz_lu, u_row_count=r.u_row_count, l_col_count=r.l_col_count,
                line_flags=r.line_flags, n_supernodes=r.n_supernodes, sn_start=_padded(r.sn_start, r.n))


def _padded(a, count):
    out = np.zeros(count, a.dtype)
    out[:a.size] = a
    return out


def _in_line_order(s, r):
    """The pool's lists, which lie as they were finished, by line: U rows, then L columns."""
    count = torch.from_numpy(np.concatenate([r.u_row_count, r.l_col_count])).cuda()
    begin = torch.from_numpy(np.concatenate([r.u_beg, r.l_beg])).cuda()
    shift = (begin - (count.cumsum(0) - count)).to(torch.int32)   # the pools here hold less than 2^31 entries
    entries = r.pool_used
    at = torch.repeat_interleave(shift, count, output_size=entries).add_(s["place"][:entries])
    torch.index_select(s["pool"], 0, at, out=s["lines"][:entries])
    return s["lines"]


def run(s):
    call = s["call"]
    if call == "noalloc":
        (b, e, a), (u, l, sn) = s["in"], s["out"]
        fills, nnz, k = gsofa_b200.symbfact_counts_noalloc(
            0, torch.cuda.current_stream().cuda_stream, s["n"], s["nnz"], b.data_ptr(), e.data_ptr(), a.data_ptr(),
            u.data_ptr(), l.data_ptr(), sn.data_ptr())
        return dict(fill_count=fills, nnz_lu=nnz, u_row_count=u, l_col_count=l, n_supernodes=k, sn_start=sn)
    if call == "counts":
        return _lines(s["ctx"].symbfact(s["matrix"], want_pattern=0))
    if call == "csr":
        r = s["ctx"].symbfact_into(s["matrix"], s["params"], s["buffers"])
        return dict(s["buffers"], fill_count=r.fill_count, nnz_lu=r.nnz_lu, n_supernodes=r.n_supernodes)
    if call == "ranges":
        with torch.cuda.stream(s["stream"]):
            r = s["ctx"].symbfact_ranges(s["matrix"], s["pool"], s["params"], out=s["buffers"])
            entries = _in_line_order(s, r)
        return dict(fill_count=r.fill_count, nnz_lu=r.nnz_lu, u_row_count=r.u_row_count, l_col_count=r.l_col_count,
                    l_row_count=r.l_row_count, n_supernodes=r.n_supernodes, sn_start=s["buffers"]["sn_start"],
                    entries=entries)
    if call == "supernodal":
        with s["ctx"].upload(s["graph"]) as m:
            r, x = s["ctx"].symbfact_supernodal(m, out=s["buffers"])
        return dict(s["buffers"], fill_count=r.fill_count, nnz_lu=r.nnz_lu, nsuper=x.nsuper)
    if call == "batch":
        rs = s["ctx"].symbfact_batch(s["mats"], s["params"])
        return _joined([_lines(r) for r in rs])
    if call == "serve":
        srv, got = s["server"], {}
        ids = []
        for g in s["graphs"]:
            rid = srv.submit(g)
            while rid is None:      # no room now: fetch what is done
                got.update((i, srv.result(i)) for i in srv.poll())
                rid = srv.submit(g)
            ids.append(rid)
        while len(got) < len(ids):
            got.update((i, srv.result(i)) for i in srv.poll())
        srv.drain()
        return _joined([_lines(got[i]) for i in ids])
    return s["ctx"].order_rcm(s["graph"])


def _joined(parts):
    """The results of many matrices, one after another."""
    return {k: np.concatenate([np.atleast_1d(p[k]) for p in parts]) for k in parts[0]}


# ----------------------------------------------------------------------------
# What a pass cannot do without


def _shape(case):
    """(lines, input entries, pattern entries): rounded laws of the generators' patterns, good to a few percent."""
    k = case["kind"]
    if k == "grid2d":
        n = case["nx"] * case["ny"]
        return n, 4.8 * n, 2.0 * n * case["nx"]
    if k == "nd3d":
        n = case["nx"] * case["ny"] * case["nz"]
        return n, 6.6 * n, 18.7 * n ** (4 / 3)
    if k == "powerlaw":
        return case["n"], 8.9 * case["n"], 0.28 * case["n"] ** 2
    if k == "bordered":
        n = 32 * case["blocks"] + 8
        return n, 5.7 * n, 20.0 * n
    n = case["count"] * (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])   # log-uniform sizes
    return n, 6.8 * n, 0.0


def work(case):
    n, nnz, entries = _shape(case)
    read = 4 * (2 * n + nnz)                       # begins, ends, ids
    if case["call"] == "order":
        return dict(bytes=read + 4 * n, flops=0)   # the permutation
    if case["call"] == "noalloc":
        return dict(bytes=read + 12 * n, flops=0)
    wrote = 13 * n                                 # two counts, a flag and a supernode start per line at most
    if case["call"] == "csr":
        wrote += 20 * n + 4 * entries
    elif case["call"] == "ranges":
        wrote += 20 * n + 4 * entries
    elif case["call"] == "supernodal":
        wrote = 28 * n + 0.16 * 4 * entries        # the structure holds one list where a supernode's lines share it
    return dict(bytes=read + wrote, flops=0)
