"""Whether a graph is symmetric is told from a sum of hashed edges. The hash takes a key that no graph can know:
here are four one-way edges whose hashes without a key (SplitMix64's finaliser of the ends) cancel. Their graph is
not symmetric, so its runs must mark as single steps do; a run that took it for symmetric would let the edges'
sources follow their targets' later moves."""
import numpy as np
import pytest

import oracle as orc
import rak_lowmem as rl

FORWARD = [(347443, 509438), (158036, 873322)]     # stored at the smaller end only
BACKWARD = [(157589, 495179), (528076, 884205)]    # stored at the larger end only
N = 900_000


def _mix64(x):
    mask = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & mask
    x = ((x ^ x >> 30) * 0xBF58476D1CE4E5B9) & mask
    x = ((x ^ x >> 27) * 0x94D049BB133111EB) & mask
    return x ^ x >> 31


def _graph():
    """Every target in a clique of five with the vertices after it, the sources with their one edge."""
    edges = []
    for source, target in FORWARD + [(b, a) for a, b in BACKWARD]:
        edges.append((source, target))
        clique = range(target, target + 5)
        edges += [(a, b) for a in clique for b in clique if a != b]
    u, v = np.array(sorted(edges)).T
    off = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=N))]).astype(np.int64)
    return rl.HostGraph(off, v.astype(np.uint32), None)


def test_the_edges_cancel_without_a_key():
    h = [[_mix64(a << 32 | b) for a, b in pairs] for pairs in (FORWARD, BACKWARD)]
    assert (sum(h[0]) - sum(h[1])) % (1 << 64) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [rl.MODE_SYNC, rl.MODE_SYNC_SPLIT])
def test_run_marks_as_steps_do(mode):
    import torch
    g = _graph()
    sources = [a for a, _ in FORWARD] + [b for _, b in BACKWARD]
    targets = [b for _, b in FORWARD] + [a for a, _ in BACKWARD]
    with rl.Context(0) as ctx:
        rg = rl.ResidentGraph(ctx, g, mode=mode)
        lab = torch.arange(N, dtype=torch.int32, device="cuda")
        aff = torch.ones(N, dtype=torch.uint8, device="cuda")
        nxt, anx = torch.empty_like(lab), torch.empty_like(aff)
        torch.cuda.synchronize()
        for k in range(5):
            rg.step(k, lab, aff, nxt, anx, mode=mode)
            lab, nxt, aff, anx = nxt, lab, anx, aff
        want = lab.cpu().numpy()
        # the targets moved on after the sources had taken their labels: the case tells the two apart
        assert any(want[s] != want[t] for s, t in zip(sources, targets))
        got, _ = ctx.lowmem(g, mode=mode, tolerance=0.0, max_iterations=5)
        rg.close()
    assert np.array_equal(got.view(np.int32), want)
    o = orc.make_opts(slots=8, rescan=1 if mode == rl.MODE_SYNC else 0, split=1 if mode == rl.MODE_SYNC_SPLIT else 0,
                      tolerance=0.0, max_iterations=5)
    assert np.array_equal(got, orc.sync_run(orc.Graph.of(g), o)[0])
