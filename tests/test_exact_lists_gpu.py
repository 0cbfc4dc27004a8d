"""The exact synchronous mode scans long lists 32 edges at a time (votes for hits, misses one by one) and short
ones edge by edge; both must equal the oracle's sequential scan, with and without the exact rescan, for lists
at the groups' limits and at remainders of 32, labels that repeat much or never, zero weights, self-loops and
duplicate edges, every slot count."""
import numpy as np
import pytest

import oracle as orc
import rak_lowmem as rl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with rl.Context(0) as c:
        yield c


def _graph(weighted, variety):
    """Centres with lists of many lengths over leaves; leaves' initial labels come from `variety` values."""
    rng = np.random.default_rng(4)
    degs = [255, 256, 257, 511, 513, 1023, 1024, 1025, 1056, 2047, 2048, 2049, 4095, 4097, 4128, 9001, 70003]
    leaves = 20000
    n = len(degs) + leaves
    u = np.concatenate([np.full(d, i) for i, d in enumerate(degs)])
    v = len(degs) + rng.integers(0, leaves, len(u))       # duplicates in the long lists
    v[::501] = u[::501]                                    # self-loops
    w = rng.uniform(0.5, 4, len(u)).astype(np.float32)
    w[::37] = 0.0
    src, dst, w = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.argsort(src, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    g = rl.HostGraph(off, dst[order].astype(np.uint32), w[order] if weighted else None)
    return g, (np.arange(n) if variety is None else rng.integers(0, variety, n)).astype(np.uint32)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("variety", [None, 5, 40])
@pytest.mark.parametrize("rescan", [0, 1])
def test_long_lists_equal_oracle(ctx, weighted, variety, rescan):
    g, q = _graph(weighted, variety)
    og = orc.Graph.of(g)
    for slots in (2, 4, 8, 16):
        o = orc.make_opts(slots=slots, rescan=rescan, tolerance=0.0, max_iterations=3)
        want, wit, _ = orc.sync_run(og, o, q)
        got, r = ctx.lowmem(g, q=q, slots=slots, mode=rl.MODE_SYNC, rescan=rescan, tolerance=0.0, max_iterations=3)
        assert r.iterations == wit
        assert np.array_equal(got, want)
