"""Device primitives through the C ABI: decoupled look-back scan, exact cut."""
import numpy as np
import pytest

import oracle
from hunyuansc25_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 31, 4095, 4096, 4097, 100000, 1 << 22, 10_000_019])
def test_scan_exclusive(ctx, n):
    import torch
    rng = np.random.default_rng(n)
    a = rng.integers(0, 50, size=n, dtype=np.int32)
    d = torch.from_numpy(a).cuda()
    out = ctx.scan_exclusive(d).cpu().numpy()
    ref = np.zeros(n + 1, np.int64)
    ref[1:] = np.cumsum(a, dtype=np.int64)
    assert np.array_equal(out.astype(np.int64), ref)


def test_scan_in_place(ctx):
    import torch
    a = np.arange(1, 300001, dtype=np.int32) % 7
    buf = torch.zeros(a.size + 1, dtype=torch.int32, device="cuda")
    buf[:-1] = torch.from_numpy(a).cuda()
    ctx.scan_exclusive(buf[:-1], buf)
    ref = np.concatenate([[0], np.cumsum(a)])
    assert np.array_equal(buf.cpu().numpy(), ref)


def test_edgecut_device(ctx):
    import torch
    g = graphs.rmat(14, 16, seed=3)
    where = (np.arange(g.nvtxs) * 2654435761 % 97).astype(np.int32)
    t = [torch.from_numpy(x).cuda() for x in (g.xadj, g.adjncy, g.adjwgt, where)]
    assert ctx.edgecut_device(t[0], t[1], t[2], t[3]) == oracle.edgecut(g, where)
    unit = graphs.Graph(g.xadj, g.adjncy, g.vwgt, np.ones_like(g.adjwgt))
    assert ctx.edgecut_device(t[0], t[1], None, t[3]) == oracle.edgecut(unit, where)


def walk_graph(degrees, seed):
    """A symmetric graph on the given target degrees (a multigraph's edges, repeats dropped)."""
    rng = np.random.default_rng(seed)
    stubs = np.repeat(np.arange(len(degrees)), degrees)
    rng.shuffle(stubs)
    stubs = stubs[: stubs.size // 2 * 2].reshape(-1, 2)
    stubs = stubs[stubs[:, 0] != stubs[:, 1]]
    e = np.unique(np.sort(stubs, 1), axis=0)
    w = rng.integers(1, 1000, e.shape[0]).astype(np.int32)
    s, d = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((d, s))
    xadj = np.zeros(len(degrees) + 1, np.int32)
    xadj[1:] = np.cumsum(np.bincount(s, minlength=len(degrees)))
    return xadj, d[order].astype(np.int32), np.concatenate([w, w])[order]


# the edge-parallel walks: empty rows in runs longer than a window of 32, hub rows over
# several warps' shares, one entry pair to several rounds of the grid
WALKS = {
    "pair": [1, 1],
    "empty_runs": [0] * 70 + [3, 5, 2] + [0] * 33 + [4] * 40 + [0] * 200,
    "hubs": [3000, 2500] + [2] * 5000 + [0] * 40 + [700] * 3 + [1] * 999,
    "odd": [5] * 1001,
    "large": [16] * 120001,
}


@pytest.mark.parametrize("name", list(WALKS))
@pytest.mark.parametrize("unit", [False, True])
def test_edgecut_walk(ctx, name, unit):
    import torch
    xadj, adj, w = walk_graph(WALKS[name], 3)
    n = xadj.size - 1
    where = np.random.default_rng(4).integers(0, 7, n).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(xadj))
    cut = int((np.ones_like(w) if unit else w)[where[rows] != where[adj]].astype(np.int64).sum()) // 2
    t = [torch.from_numpy(a).cuda() for a in (xadj, adj, w, where)]
    torch.cuda.synchronize()
    assert ctx.edgecut_device(t[0], t[1], None if unit else t[2], t[3]) == cut


def _path_with_gaps(m, gap, every):
    """A path over m vertices, `gap` vertices without edges before every `every`-th of them."""
    at = np.arange(m) + gap * (np.arange(m) // every)
    n = int(at[-1]) + 1 + gap
    xadj = np.zeros(n + 1, np.int32)
    xadj[at + 1] = 2
    xadj[at[0] + 1] = xadj[at[-1] + 1] = 1
    adj = np.stack([np.concatenate([[-1], at[:-1]]), np.concatenate([at[1:], [-1]])], 1).ravel()[1:-1]
    return np.cumsum(xadj, dtype=np.int32), adj.astype(np.int32)


# runs of empty rows that end at, before and after the walks' windows, between single rows
# and between groups of them
@pytest.mark.parametrize("gap", [31, 32, 63, 64, 65, 95, 96, 97, 129, 1000, 70001])
@pytest.mark.parametrize("every", [1, 7, 40])
def test_walks_over_runs_of_empty_rows(ctx, gap, every):
    import torch

    import hunyuansc25_b200 as hp
    xadj, adj = _path_with_gaps(min(300, max(3 * every, 2_000_000 * every // gap)), gap, every)
    n = xadj.size - 1
    rows = np.repeat(np.arange(n), np.diff(xadj))
    where = np.random.default_rng(gap).integers(0, 5, n).astype(np.int32)
    t = [torch.from_numpy(a).cuda() for a in (xadj, adj, where)]
    torch.cuda.synchronize()
    assert ctx.edgecut_device(t[0], t[1], None, t[2]) == int((where[rows] != where[adj]).sum()) // 2
    # the validation: accepted as it is, refused with one entry that has no reverse
    if n < 20000:
        ctx.partition(xadj, adj, 2)
    bad = adj.copy()
    bad[-1] = rows[0] if rows[0] != bad[-1] else rows[2]
    with pytest.raises(hp.HpError):
        ctx.partition(xadj, bad, 2)


def test_long_run_of_empty_rows_is_passed_quickly(ctx):
    """Eight million vertices without edges between two rows cost the edge cut and the
    validation no walk over them (window by window they take over 80 ms)."""
    import time

    import torch

    import hunyuansc25_b200 as hp
    xadj, adj = _path_with_gaps(2000, 1 << 23, 1000)
    n = xadj.size - 1
    t = [torch.from_numpy(a).cuda() for a in (xadj, adj)]
    where = torch.zeros(n, dtype=torch.int32, device="cuda")
    adj[-1] = 5   # no reverse: refused right after the validation
    bad = torch.from_numpy(adj).cuda()
    part = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def refused():
        with pytest.raises(hp.HpError):
            ctx.partition_device(t[0], bad, 2, part=part)

    for call in (lambda: ctx.edgecut_device(t[0], t[1], None, where), refused):
        best = 1e9
        for _ in range(4):
            t0 = time.perf_counter()
            call()
            best = min(best, time.perf_counter() - t0)
        assert best < 0.03, best


@pytest.mark.parametrize("at", [0, 31, 32, 127, 128, 129, 500])
def test_validation_of_unsorted_rows(ctx, at):
    """A row that is not ascending at one place is accepted, one that lists a neighbour twice
    (there, or far apart) is refused, wherever the place falls in a warp's batches."""
    import hunyuansc25_b200 as hp
    n = 700
    xadj = np.arange(0, n * (n - 1) + 1, n - 1).astype(np.int32)
    adj = np.stack([np.delete(np.arange(n), v) for v in range(n)]).astype(np.int32)
    v = 3 + at
    ok = adj.copy()
    ok[v, [at, at + 1]] = ok[v, [at + 1, at]]
    part, cut = ctx.partition(xadj, ok.ravel(), 2)
    ref, rcut = ctx.partition(xadj, adj.ravel(), 2)
    assert cut == rcut
    for other in (at + 1, (at + 300) % (n - 1)):
        bad = adj.copy()
        bad[v, other] = bad[v, at]
        with pytest.raises(hp.HpError):
            ctx.partition(xadj, bad.ravel(), 2)
