"""Synchronous runs find an iteration's active vertices either from marks (every move flags the mover's
neighbours, inc/rakCuda.hxx:95-103) or, on symmetric graphs where most vertices move, by looking for a
neighbour that moved. Single steps always mark, so a run of k iterations must equal k steps: labels and
counts of moved vertices, at every k, on symmetric graphs, on graphs that lack one reverse edge, with
duplicate edges and self-loops, from sparse initial flags, and in batches where one graph is asymmetric."""
import numpy as np
import pytest

import oracle as orc
import rak_lowmem as rl

pytestmark = pytest.mark.gpu

LAYOUT = dict(lane_max=8, hub_min=64, hub_chunk=32)   # every work region at small degrees


@pytest.fixture(scope="module")
def ctx():
    with rl.Context(0) as c:
        yield c


def _csr(n, u, v):
    order = np.lexsort((v, u))
    u, v = u[order], v[order]
    off = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.int64)
    return rl.HostGraph(off, v.astype(np.uint32), None)


def _graph(kind, seed=3):
    rng = np.random.default_rng(seed)
    n = 1501
    a = rng.integers(0, n, 6000)
    b = np.where(rng.random(6000) < 0.8, (a // 50) * 50 + rng.integers(0, 50, 6000), rng.integers(0, n, 6000)) % n
    a, b = np.concatenate([a, np.zeros(300, int)]), np.concatenate([b, rng.integers(1, n, 300)])   # a split vertex
    u, v = np.concatenate([a, b]), np.concatenate([b, a])
    if kind == "one_way":          # one edge without its reverse
        u, v = u[1:], v[1:]
    if kind == "loops":
        x = rng.integers(0, n, 200)
        u, v = np.concatenate([u, x, x]), np.concatenate([v, x, x])
    if kind == "directed":
        u, v = a, b
    return _csr(n, u, v)


@pytest.mark.parametrize("kind", ["symmetric", "one_way", "loops", "directed"])
@pytest.mark.parametrize("mode", [rl.MODE_SYNC, rl.MODE_SYNC_SPLIT])
@pytest.mark.parametrize("slots", [8, 1])
def test_run_equals_steps(ctx, kind, mode, slots):
    import torch
    g = _graph(kind)
    n = g.n
    opts = dict(slots=slots, mode=mode, **LAYOUT)
    rg = rl.ResidentGraph(ctx, g, **opts)
    lab = torch.arange(n, dtype=torch.int32, device="cuda")
    aff = torch.ones(n, dtype=torch.uint8, device="cuda")
    nxt, anx = torch.empty_like(lab), torch.empty_like(aff)
    out = torch.empty_like(lab)
    torch.cuda.synchronize()
    total = 0
    for k in range(1, 13):
        moved = rg.step(k - 1, lab, aff, nxt, anx, **opts)
        total += moved
        r = rg.run(out, tolerance=0.0, max_iterations=k, **opts)
        assert torch.equal(out, nxt)
        if r.iterations == k:
            assert r.moved_vertices == total and r.changed_last == moved
        lab, nxt, aff, anx = nxt, lab, anx, aff
        if moved == 0:
            break


@pytest.mark.parametrize("kind", ["symmetric", "one_way"])
def test_sparse_initial_flags(ctx, kind):
    g = _graph(kind)
    flags = np.zeros(g.n, np.uint8)
    flags[::97] = 1
    import torch
    opts = dict(slots=8, mode=rl.MODE_SYNC_SPLIT, **LAYOUT)
    rg = rl.ResidentGraph(ctx, g, **opts)
    lab = torch.arange(g.n, dtype=torch.int32, device="cuda")
    aff = torch.from_numpy(flags).cuda()
    nxt, anx = torch.empty_like(lab), torch.empty_like(aff)
    torch.cuda.synchronize()
    for k in range(1, 9):
        rg.step(k - 1, lab, aff, nxt, anx, **opts)
        got, _ = ctx.lowmem(g, flags=flags, tolerance=0.0, max_iterations=k, **opts)
        assert np.array_equal(got, nxt.cpu().numpy().view(np.uint32))
        lab, nxt, aff, anx = nxt, lab, anx, aff


@pytest.mark.parametrize("mode", [rl.MODE_SYNC, rl.MODE_SYNC_SPLIT])
@pytest.mark.parametrize("kinds", [["symmetric", "loops"], ["symmetric", "one_way", "loops"]])
def test_batch_equals_graphs_alone(ctx, mode, kinds):
    import torch
    graphs = [_graph(k, seed=5 + i) for i, k in enumerate(kinds)]
    b = rl.Batch(ctx, rl.HostBatch.concat(graphs), mode=mode, slots=8, **LAYOUT)
    out = torch.empty(b.n, dtype=torch.int32, device="cuda")
    b.launch(out, mode=mode, slots=8, **LAYOUT)
    its, _ = b.results()
    first = 0
    for g, it in zip(graphs, its):
        want, wit = _oracle(g, mode)
        assert wit == it
        assert np.array_equal(out[first:first + g.n].cpu().numpy().view(np.uint32), want)
        first += g.n


def _oracle(g, mode):
    o = orc.make_opts(slots=8, rescan=1 if mode == rl.MODE_SYNC else 0, split=1 if mode == rl.MODE_SYNC_SPLIT else 0,
                      layout=(LAYOUT["lane_max"], LAYOUT["hub_min"], LAYOUT["hub_chunk"]))
    return orc.sync_run(orc.Graph.of(g), o)[:2]
