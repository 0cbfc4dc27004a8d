"""Long edge chains are scanned by a whole block (one thread per slot) where the graph is small and by a
warp where it is large. The line goes by the edges of the launch, so a graph in a batch beside a large
one is scanned by warps, and alone by blocks: its labels and iteration count must be the same bit for bit,
for degrees around the lane groups' and split vertices' limits, every slot count, weights and unit weights."""
import numpy as np
import pytest

import oracle as orc
import rak_lowmem as rl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with rl.Context(0) as c:
        yield c


def _ladder(weighted):
    """Centres whose degrees sit around 8, 32, 256 and its multiples, a region-1 vertex and a split one."""
    rng = np.random.default_rng(2)
    degs = [7, 8, 9, 31, 32, 33, 63, 200, 255, 256, 257, 512, 513, 1025, 2049, 4097, 9000, 20011, 65536, 65537, 70001]
    leaves = 72000
    n = len(degs) + leaves
    u = np.concatenate([np.full(d, i) for i, d in enumerate(degs)])
    v = len(degs) + np.concatenate([rng.choice(leaves, d, replace=False) for d in degs])
    a = rng.integers(0, leaves, 60000)
    b = np.minimum(leaves - 1, a // 40 * 40 + rng.integers(0, 40, 60000))
    u, v = np.concatenate([u, len(degs) + a]), np.concatenate([v, len(degs) + b])
    w = rng.uniform(1, 10, len(u)).astype(np.float32)
    src, dst, w = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.lexsort((dst, src))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    return rl.HostGraph(off, dst[order].astype(np.uint32), w[order] if weighted else None)


def _ring(weighted, n=2_200_000, reach=8):
    """A ring of 2 * reach neighbours: 35 million edges, which put the batch above the line."""
    at = np.arange(n, dtype=np.int64)
    tgt = np.empty((n, 2 * reach), np.uint32)
    for j in range(reach):
        tgt[:, 2 * j] = (at + j + 1) % n
        tgt[:, 2 * j + 1] = (at - j - 1) % n
    return rl.HostGraph(np.arange(n + 1, dtype=np.int64) * 2 * reach, tgt.reshape(-1),
                        np.ones(n * 2 * reach, np.float32) if weighted else None)


@pytest.mark.parametrize("weighted", [False, True])
def test_block_scan_equals_warp_scan(ctx, weighted):
    import torch
    g, ring = _ladder(weighted), _ring(weighted)
    both = rl.Batch(ctx, rl.HostBatch.concat([g, ring]))
    out = torch.empty(both.n, dtype=torch.int32, device="cuda")
    for slots in (2, 4, 8, 16):
        opts = dict(slots=slots, mode=rl.MODE_SYNC_SPLIT, max_iterations=6)
        alone, r = ctx.lowmem(g, **opts)
        both.launch(out, **opts)
        its, _ = both.results()
        assert its[0] == r.iterations
        assert np.array_equal(out[:g.n].cpu().numpy().view(np.uint32), alone)
    o = orc.make_opts(slots=8, split=1, max_iterations=6)
    want, wit, _ = orc.sync_run(orc.Graph.of(g), o)
    got, r = ctx.lowmem(g, slots=8, mode=rl.MODE_SYNC_SPLIT, max_iterations=6)
    assert r.iterations == wit and np.array_equal(got, want)
