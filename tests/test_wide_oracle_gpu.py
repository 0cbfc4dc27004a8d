"""Long edge chains at every slot count against the oracle's split run: 2, 4, 8 and 16 slots give a chain 2 to 16
threads of a block, 128 to 16 chains at a time, so the longest lists are checked independently at each, alone and in
a batch beside a large graph (where the lists of more than 17472 edges are still scanned by blocks)."""
import numpy as np
import pytest

import oracle as orc
import rak_lowmem as rl
from test_wide_items_gpu import _ladder, _ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
def test_long_lists_at_every_slot_count(weighted):
    import torch
    g, ring = _ladder(weighted), _ring(weighted)
    og = orc.Graph.of(g)
    with rl.Context(0) as ctx:
        both = rl.Batch(ctx, rl.HostBatch.concat([g, ring]))
        out = torch.empty(both.n, dtype=torch.int32, device="cuda")
        for slots in (2, 4, 8, 16):
            opts = dict(slots=slots, mode=rl.MODE_SYNC_SPLIT, max_iterations=6)
            want, wit, _ = orc.sync_run(og, orc.make_opts(slots=slots, split=1, max_iterations=6))
            got, r = ctx.lowmem(g, **opts)
            assert r.iterations == wit and np.array_equal(got, want), slots
            both.launch(out, **opts)
            its, _ = both.results()
            assert its[0] == wit
            assert np.array_equal(out[:g.n].cpu().numpy().view(np.uint32), want), slots
        both.close()
