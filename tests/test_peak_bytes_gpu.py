"""peak_device_bytes is all device memory a call held: the scratch that its context keeps from an earlier call
too."""
import numpy as np
import pytest

import rak_lowmem as rl

pytestmark = pytest.mark.gpu


def test_kept_scratch_is_counted():
    import torch
    g = rl.gen_rmat(8, 8, seed=1)
    off = torch.from_numpy(g.offsets).cuda()
    tgt = torch.from_numpy(g.targets.view(np.int32)).cuda()
    csr = rl.device_csr(off, tgt, None)
    out = torch.empty(g.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def calls(ctx):
        rg = rl.ResidentGraph(ctx, csr, mode=rl.MODE_SYNC_SPLIT)
        run = rg.run(out, mode=rl.MODE_SYNC_SPLIT, compute_modularity=1).peak_device_bytes
        rg.close()
        return [run, ctx.lowmem_device(csr, out, mode=rl.MODE_SYNC_SPLIT).peak_device_bytes,
                ctx.lowmem(g, mode=rl.MODE_SYNC_SPLIT)[1].peak_device_bytes]

    with rl.Context(0) as ctx:
        before = calls(ctx)
    with rl.Context(0) as ctx:
        n = 2_000_000     # 8 bytes a vertex, kept
        ctx.modularity(rl.HostGraph(np.zeros(n + 1, np.int64), np.zeros(0, np.uint32)), np.zeros(n, np.uint32))
        after = calls(ctx)
    assert all(b < 1 << 20 for b in before)
    assert all(a >= 8 * n and a - b >= 8 * n - (1 << 20) for a, b in zip(after, before))


@pytest.mark.parametrize("hub_min", [65536, 1 << 30])
def test_small_chunks_of_no_split_vertex_take_no_room(hub_min):
    """A one-shot call makes room for split vertices' tables before it knows of any: not for 2 bytes an edge. With
    split vertices, more of them than it has room for, the call works all the same."""
    g = rl.gen_rmat(14, 32, seed=3)
    with rl.Context(0) as ctx:
        _, usual = ctx.lowmem(g, mode=rl.MODE_SYNC_SPLIT)
        _, small = ctx.lowmem(g, mode=rl.MODE_SYNC_SPLIT, hub_min=hub_min, hub_chunk=32)
        # at most a label array more
        assert small.peak_device_bytes <= usual.peak_device_bytes + 4 * g.n + 4096
        opts = dict(mode=rl.MODE_SYNC_SPLIT, hub_min=256, hub_chunk=32)
        labels, _ = ctx.lowmem(g, **opts)
        import torch
        rg, out = rl.ResidentGraph(ctx, g, **opts), torch.empty(g.n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rg.run(out, **opts)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), labels)
        rg.close()
