"""Weighted modularity takes the totals of short rows 32 edges at a time. A row's total holds its own edges only:
rows between two of weight +A and -A keep their totals although A is 2^60 times larger. The two large rows lie 16
apart, so that the warp's sum of the rows' totals cancels them first, and each row is a community of its own."""
import numpy as np
import pytest

import rak_lowmem as rl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_row", [1, 2, 3])
@pytest.mark.parametrize("bits", [32, 64])
def test_small_rows_between_large_ones(per_row, bits):
    import torch
    n, big = 512, 2.0 ** 60                  # the rows with edges are the first warp's of eight
    deg = np.where(np.arange(n) < 32, per_row, 0)
    deg[[0, 16]] = 1
    off = np.concatenate([[0], np.cumsum(deg)])
    m = int(off[-1])
    wt = np.arange(1, m + 1).astype(np.float32)
    wt[off[0]], wt[off[16]] = big, -big
    src = np.repeat(np.arange(n), deg)
    tgt = (src + 1) % n                      # no edge inside a community
    small = [int(wt[off[r]:off[r + 1]].sum()) for r in range(32) if r not in (0, 16)]
    total = sum(small)                       # exact: whole numbers below 2^24
    want = -(2 * big * big + sum(s * s for s in small)) / total ** 2
    d = [torch.from_numpy(x).cuda() for x in (off.astype(np.int64 if bits == 64 else np.int32), tgt.astype(np.int32), wt,
                                              np.arange(n, dtype=np.int32))]
    torch.cuda.synchronize()
    with rl.Context(0) as ctx:
        got = ctx.modularity(rl.device_csr(d[0], d[1], d[2]), d[3])
    # a square, a sum of 32 squares, a square, a quotient: each rounded once
    assert abs(got / want - 1) <= 40 * 2.0 ** -53
