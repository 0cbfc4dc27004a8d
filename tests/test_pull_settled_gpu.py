"""Pulled iterations of the synchronous modes where long lists have settled: a vertex with many neighbours, none
of which moves any more, beside pairs that swap labels for ever. An iteration that pulls must not read the settled
list again and again: it may cost no more than a few times what marking costs. The same graph with one edge that
lacks its reverse is never pulled; labels and counts of both must be the same. In a batch the settled graph
finishes, and its split vertex's chunks take no further part."""
import numpy as np
import pytest

import rak_lowmem as rl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with rl.Context(0) as c:
        yield c


def _csr(n, u, v):
    order = np.lexsort((v, u))
    off = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.int64)
    return rl.HostGraph(off, v[order].astype(np.uint32), None)


def _star(leaves, first=0):
    """A centre and its leaves in cliques of four: the cliques settle in a few iterations, then the centre does."""
    at = first + 1 + np.arange(leaves)
    base = at[::4]
    pairs = [(base + i, base + j) for i in range(4) for j in range(i)]
    return np.concatenate([np.full(leaves, first)] + [p[0] for p in pairs]), np.concatenate([at] + [p[1] for p in pairs])


def _swapping(pairs, first):
    at = first + 2 * np.arange(pairs)
    return at, at + 1


def _both_ways(u, v):
    return np.concatenate([u, v]), np.concatenate([v, u])


def _star_and_pairs(leaves, one_way):
    """Pairs hold half of the edges. The last two vertices: an edge without its reverse, or none."""
    su, sv = _star(leaves)
    pu, pv = _swapping(len(su), leaves + 1)
    n = leaves + 1 + 2 * len(su) + 2
    u, v = _both_ways(np.concatenate([su, pu]), np.concatenate([sv, pv]))
    if one_way:
        u, v = np.append(u, n - 2), np.append(v, n - 1)
    return _csr(n, u, v)


@pytest.mark.parametrize("leaves", [4096, 60000, 65536, 65540, 400000])   # region 1 up to 65536 edges, then split
@pytest.mark.parametrize("mode", [rl.MODE_SYNC, rl.MODE_SYNC_SPLIT])
def test_settled_list_beside_moving_pairs(ctx, leaves, mode):
    import torch
    ms, labels, moved, edges = [], [], [], []
    for one_way in (False, True):
        g = _star_and_pairs(leaves, one_way)
        rg = rl.ResidentGraph(ctx, g, mode=mode)
        out = torch.empty(g.n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        took = []
        for _ in range(3):
            r = rg.run(out, mode=mode, tolerance=0.0, max_iterations=30)
            assert r.iterations == 30
            took.append(r.loop_ms)
        ms.append(min(took))
        labels.append(out.cpu().numpy()[:g.n - 2])
        moved.append(r.moved_vertices)
        edges.append(r.moved_edges)
    assert np.array_equal(labels[0], labels[1])
    assert moved[0] in (moved[1], moved[1] - 1)   # the one-way edge moves its vertex once
    assert edges[0] in (edges[1], edges[1] - 1)
    # 30 iterations; 0.2 ms: the grid barriers and launch jitter of either side
    assert ms[0] <= 3 * ms[1] + 0.2, ms


@pytest.mark.parametrize("mode", [rl.MODE_SYNC, rl.MODE_SYNC_SPLIT])
@pytest.mark.parametrize("layout", [{}, dict(lane_max=8, hub_min=64, hub_chunk=32)])
def test_batch_with_a_finished_graph(ctx, mode, layout):
    import torch
    settles = _csr(401, *_both_ways(*_star(400)))
    su, sv = _star(700)
    pu, pv = _swapping(3000, 701)
    moving = _csr(701 + 6000, *_both_ways(np.concatenate([su, pu]), np.concatenate([sv, pv])))
    graphs = [settles, moving, settles]
    opts = dict(mode=mode, tolerance=0.0, max_iterations=25, **layout)
    b = rl.Batch(ctx, rl.HostBatch.concat(graphs), **opts)
    out = torch.empty(b.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        b.launch(out, **opts)
        its, _ = b.results()
        first = 0
        for g, it in zip(graphs, its):
            want, r = ctx.lowmem(g, **opts)
            assert r.iterations == it
            assert np.array_equal(out[first:first + g.n].cpu().numpy().view(np.uint32), want)
            first += g.n
    assert its[0] < its[1] == 25
