"""FP64 modularity on the device against the same sums in numpy, at row lengths, row counts and label
patterns where the split of rows and edges over warps can go wrong (empty stretches, hubs, one edge)."""
import numpy as np
import pytest

import rak_lowmem as rl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with rl.Context(0) as c:
        yield c


def _modularity(off, tgt, wt, c):
    src = np.repeat(np.arange(len(off) - 1), np.diff(off))
    w = np.ones(len(tgt)) if wt is None else wt.astype(np.float64)
    tot = w.sum()
    per = np.bincount(c[src], weights=w, minlength=len(off) - 1)
    return w[c[src] == c[tgt]].sum() / tot - (per * per).sum() / (tot * tot)


def _degrees(kind, rng):
    if kind == "one_edge":
        return np.array([0] * 70 + [1] + [0] * 41)
    if kind == "hub":
        d = rng.integers(0, 4, 3001)
        d[1500] = 200003
        return d
    if kind == "empty_stretch":
        d = np.zeros(50007, np.int64)
        d[[0, 3, 25000, 50006]] = [5, 1, 33, 2]
        return d
    if kind == "one_row":
        return np.array([4097])
    if kind == "short":
        return rng.integers(0, 3, 1025)
    return rng.integers(0, 130, 4099)   # mixed


@pytest.mark.parametrize("kind", ["one_edge", "hub", "empty_stretch", "one_row", "short", "mixed"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("bits", [32, 64])
def test_modularity_rows_and_labels(ctx, kind, weighted, bits):
    import torch
    rng = np.random.default_rng(7)
    deg = _degrees(kind, rng)
    n, m = len(deg), int(deg.sum())
    off = np.concatenate([[0], np.cumsum(deg)])
    tgt = rng.integers(0, n, m)
    wt = rng.uniform(1, 10, m).astype(np.float32) if weighted else None
    d_off = torch.from_numpy(off.astype(np.int64 if bits == 64 else np.int32)).cuda()
    d_tgt = torch.from_numpy(tgt.astype(np.int32)).cuda()
    d_wt = None if wt is None else torch.from_numpy(wt).cuda()
    for c in (np.zeros(n, np.int64), np.arange(n), np.arange(n) // 50, rng.integers(0, max(1, n // 3), n)):
        d_c = torch.from_numpy(c.astype(np.int32)).cuda()
        torch.cuda.synchronize()
        q = ctx.modularity(rl.device_csr(d_off, d_tgt, d_wt), d_c)
        # three sums of at most m terms, each rounded once: m * 2^-53 relative; the terms are below 1
        assert abs(q - _modularity(off, tgt, wt, c)) <= 4 * max(m, 16) * 2.0 ** -53


def test_modularity_checks_targets_at_any_alignment(ctx):
    """The target check reads 16-byte vectors: every position of a bad target, whatever the array's start, is found."""
    import torch
    n, m = 1000, 77
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = m
    c = torch.zeros(n, dtype=torch.int32, device="cuda")
    for shift in range(4):
        room = torch.zeros(m + 4, dtype=torch.int32, device="cuda")
        tgt = room[shift:shift + m]
        torch.cuda.synchronize()
        ctx.modularity(rl.device_csr(off, tgt), c)
        for at in (0, 1, 2, 3, 4, 40, m - 4, m - 2, m - 1):
            tgt[at] = n
            torch.cuda.synchronize()
            with pytest.raises(rl.RakError):
                ctx.modularity(rl.device_csr(off, tgt), c)
            tgt[at] = 0
