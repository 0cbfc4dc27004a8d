"""A context keeps device scratch of up to 64 MiB for its next call (modularity, single steps, the CSR check):
calls of growing and shrinking sizes, above the limit too, interleaved with runs, and contexts on two threads,
give the same results as calls on fresh contexts."""
import threading

import numpy as np
import pytest

import rak_lowmem as rl

pytestmark = pytest.mark.gpu


def _calls(ctx, graphs):
    import torch
    out = []
    for g in graphs:
        labels, r = ctx.lowmem(g, mode=rl.MODE_SYNC_SPLIT, max_iterations=4, compute_modularity=1)
        q = ctx.modularity(g, labels)
        rg = rl.ResidentGraph(ctx, g, mode=rl.MODE_SYNC_SPLIT)
        lab = torch.arange(g.n, dtype=torch.int32, device="cuda")
        aff = torch.ones(g.n, dtype=torch.uint8, device="cuda")
        nxt, anx = torch.empty_like(lab), torch.empty_like(aff)
        torch.cuda.synchronize()
        moved = rg.step(0, lab, aff, nxt, anx, mode=rl.MODE_SYNC_SPLIT)
        res = torch.empty_like(lab)
        torch.cuda.synchronize()
        again = rg.run(res, mode=rl.MODE_SYNC_SPLIT, max_iterations=4, repeat=2, compute_modularity=1)
        assert np.array_equal(res.cpu().numpy().view(np.uint32), labels)
        assert q == r.modularity == again.modularity or abs(q - again.modularity) < 1e-12
        out.append((labels, r.iterations, round(q, 12), moved))
    return out


def test_scratch_of_any_size():
    big = rl.HostGraph(np.arange(9_000_001, dtype=np.int64) // 2, (np.arange(4_500_000, dtype=np.uint32) * 2 + 1) % 9_000_000)
    graphs = [rl.gen_rmat(8, 8, seed=1), rl.gen_rmat(14, 16, seed=2, w_lo=1.0, w_hi=4.0), big, rl.gen_rmat(6, 4, seed=3),
              rl.gen_sbm(3000, 10, seed=4), rl.gen_rmat(17, 8, seed=5)]
    want = []
    for g in graphs:
        with rl.Context(0) as c:
            want += _calls(c, [g])
    with rl.Context(0) as c:
        for order in (range(len(graphs)), reversed(range(len(graphs)))):
            for i in order:
                got = _calls(c, [graphs[i]])[0]
                assert np.array_equal(got[0], want[i][0]) and got[1:] == want[i][1:]
    small = [i for i in range(len(graphs)) if i != 2]
    errors = []

    def work():
        try:
            with rl.Context(0) as c:
                for i in small:
                    got = _calls(c, [graphs[i]])[0]
                    assert np.array_equal(got[0], want[i][0]) and got[1:] == want[i][1:]
        except BaseException as e:   # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work) for _ in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
