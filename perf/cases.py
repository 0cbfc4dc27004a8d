"""The work that users of this library have it do, through its public Python entry points.

Families and sizes are those of the repository's benchmark and tests: symmetric R-MAT graphs
(0.57, 0.19, 0.19, 0.05), planted-partition SBM graphs (average degree 16, p_in/p_out 20) and road-like
2D lattices (5% of the edges deleted, 1% shortcuts). Every input is made on the GPU from the seed alone.

What a pass returns. The synchronous modes are deterministic, so their cases return the whole membership.
Asynchronous runs (the default) update labels in place and end in other labels each time, so what is
reproducible about them is the FP64 modularity of the communities they find, which the run itself
computes (compute_modularity). One run's modularity is a noisy number; these cases therefore run several
independent graphs one after the other, as a program over a set of graphs does, and return one
modularity for each graph.
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "rak-lowmem-communities-cuda_b200"))

SYNC, SPLIT = 1, 2       # rak_mode values (0: asynchronous, the default)
ASYNC = 0


# ---- the cases -----------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one little graph in a latency-critical loop, no device allocation
        {"name": "noalloc_small", "kind": "noalloc", "family": "rmat", "n": 4096, "degree": 32, "weighted": False, "bits": 64,
         "slots": 8, "mode": SPLIT},
        # the exact synchronous mode (bit-identical to the reference's CPU rules), on the graph of the
        # reference's own CPU comparison (scale 16, edge factor 16)
        {"name": "exact_rmat16", "kind": "resident", "family": "rmat", "n": 65536, "degree": 32, "weighted": False, "bits": 32,
         "slots": 8, "mode": SYNC},
        # the drop-in call on a host graph: upload, plan, run, membership back (float weights, int32 CSR)
        {"name": "host_call", "kind": "host", "family": "rmat", "n": 131072, "degree": 32, "weighted": True, "bits": 32,
         "slots": 8, "mode": SPLIT},
        # reproducible communities of a weighted graph that stays resident (edge factor 32, U[1,10))
        {"name": "split_weighted", "kind": "resident", "family": "rmat", "n": 1 << 20, "degree": 64, "weighted": True,
         "bits": 32, "slots": 8, "mode": SPLIT},
        # the largest graph here: the headline family (edge factor 16, unit weights, int64 offsets)
        {"name": "split_large", "kind": "resident", "family": "rmat", "n": 1 << 24, "degree": 32, "weighted": False, "bits": 64,
         "slots": 8, "mode": SPLIT},
        # the default mode on the graphs of the serving load's large requests (scale 22, edge factor 16)
        {"name": "async_rmat22", "kind": "set", "family": "rmat", "n": 1 << 22, "degree": 32, "weighted": False, "bits": 64,
         "slots": 8, "graphs": 8},
        # the default mode on weighted graphs (edge factor 32, U[1,10), int32 CSR); on smaller weighted
        # R-MAT graphs some runs end in one community, others not
        {"name": "async_weighted", "kind": "set", "family": "rmat", "n": 1 << 22, "degree": 64, "weighted": True, "bits": 32,
         "slots": 8, "graphs": 4},
        # the default mode on road-like lattices of an odd size
        {"name": "async_lattice", "kind": "set", "family": "lattice", "n": 2047 * 2049, "degree": 4, "weighted": False,
         "bits": 32, "slots": 8, "graphs": 8},
        # the Boyer-Moore variant (one slot) on planted communities
        {"name": "async_bm_sbm", "kind": "set", "family": "sbm", "n": 300007, "degree": 16, "weighted": False, "bits": 32,
         "slots": 1, "graphs": 8},
        # many uneven graphs in one persistent launch, replayed from its CUDA graph
        {"name": "batch_mix", "kind": "batch", "family": "mix", "n": 1 << 23, "graphs": 256, "weighted": False, "bits": 64,
         "slots": 8, "mode": SPLIT, "degree": 24},
        # the request loop: graphs that are resident on the device, submitted at once
        {"name": "serve_mix", "kind": "serve", "family": "mix", "n": 1 << 21, "graphs": 96, "weighted": False, "bits": 64,
         "slots": 8, "mode": SPLIT, "degree": 24},
        # FP64 modularity of a given partition of a weighted graph
        {"name": "modularity", "kind": "modularity", "family": "rmat", "n": 1 << 21, "degree": 32, "weighted": True, "bits": 32},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["noalloc", "resident", "resident", "exact", "host", "set", "set", "set", "batch", "serve",
                       "modularity"])
    weighted = rng.random() < 0.4
    bits = rng.choice([32, 64])
    if kind == "noalloc":
        return {"kind": kind, "family": rng.choice(["rmat", "sbm"]), "n": _log(rng, 1000, 50000),
                "degree": rng.choice([8, 16, 32]), "weighted": weighted, "bits": bits, "slots": 8, "mode": SPLIT}
    if kind == "exact":
        return {"kind": "resident", "family": rng.choice(["rmat", "sbm"]), "n": _log(rng, 4000, 100000),
                "degree": rng.choice([16, 32]), "weighted": weighted, "bits": bits, "slots": 8, "mode": SYNC}
    if kind == "host":
        return {"kind": kind, "family": rng.choice(["rmat", "sbm"]), "n": _log(rng, 10000, 500000),
                "degree": rng.choice([16, 32]), "weighted": weighted, "bits": bits, "slots": 8, "mode": SPLIT}
    if kind == "resident":
        return {"kind": kind, "family": rng.choice(["rmat", "rmat", "sbm"]), "n": _log(rng, 30000, 2000000 if weighted else 8000000),
                "degree": rng.choice([16, 32]), "weighted": weighted, "bits": bits, "slots": rng.choice([8, 8, 8, 4]),
                "mode": SPLIT}
    if kind == "set":
        family = rng.choice(["rmat", "lattice", "sbm"])
        weighted = weighted and family == "rmat"
        return {"kind": kind, "family": family, "n": _log(rng, 2500000 if weighted else 200000, 4000000),
                "degree": {"rmat": 64 if weighted else 32, "lattice": 4, "sbm": 16}[family], "weighted": weighted,
                "bits": bits, "slots": 8 if family == "rmat" else rng.choice([8, 8, 1]), "graphs": 4 if weighted else 8}
    if kind == "modularity":
        return {"kind": kind, "family": rng.choice(["rmat", "sbm", "lattice"]), "n": _log(rng, 20000, 2000000),
                "degree": 16, "weighted": weighted, "bits": bits}
    return {"kind": kind, "family": "mix", "n": _log(rng, 1 << 18, 1 << 22), "graphs": rng.choice([32, 64, 128]),
            "weighted": weighted, "bits": 64, "slots": 8, "mode": SPLIT, "degree": 24}


# ---- graphs, made on the GPU ----------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _csr(u, v, n, weighted, bits, gen):
    """Symmetric, duplicate-free CSR of the undirected pairs (u, v); the weight of a pair, the same both
    ways, is uniform in [1, 10)."""
    keep = u != v
    lo, hi = torch.minimum(u, v)[keep], torch.maximum(u, v)[keep]
    key = torch.unique(lo * n + hi)
    lo, hi = key // n, key % n
    w = torch.rand(key.numel(), device="cuda", generator=gen) * 9 + 1 if weighted else None
    del key
    both, order = torch.sort(torch.cat([lo * n + hi, hi * n + lo]))
    w = torch.cat([w, w])[order] if weighted else None
    del order, lo, hi
    src = both // n
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return off if bits == 64 else off.int(), (both - src * n).int(), w


def _graph(family, n, degree, weighted, bits, gen):
    if family == "rmat":    # ids in the recursion's order, spread over n vertices
        scale, m = max(1, (n - 1).bit_length()), n * degree // 2
        u = torch.zeros(m, dtype=torch.int64, device="cuda")
        v = torch.zeros(m, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = torch.rand(m, device="cuda", generator=gen)
            u = u * 2 + (r >= 0.76)
            v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        u, v = u * n >> scale, v * n >> scale
    elif family == "sbm":   # blocks of about 1000 vertices (at least 8 of them), p_in / p_out = 20
        k, m = max(8, n // 1000), n * degree // 2
        s = n / k
        inside = 20 * (s - 1) / (20 * (s - 1) + (n - s))
        u = torch.randint(n, (m,), device="cuda", generator=gen)
        b = u * k // n
        first, last = -(-b * n // k), -(-(b + 1) * n // k)
        r = torch.rand(m, dtype=torch.float64, device="cuda", generator=gen)
        v = torch.where(torch.rand(m, device="cuda", generator=gen) < inside, first + (r * (last - first)).long(),
                        (r * n).long())
    else:                   # lattice
        h = max(2, int(round(n ** 0.5)))
        width = max(2, n // h)
        n = width * h
        at = torch.arange(n, device="cuda").view(h, width)
        u = torch.cat([at[:, :-1].reshape(-1), at[:-1].reshape(-1)])
        v = torch.cat([at[:, 1:].reshape(-1), at[1:].reshape(-1)])
        keep = torch.rand(u.numel(), device="cuda", generator=gen) >= 0.05
        extra = torch.randint(n, (2, u.numel() // 100), device="cuda", generator=gen)
        u, v = torch.cat([u[keep], extra[0]]), torch.cat([v[keep], extra[1]])
    return _csr(u, v, n, weighted, bits, gen)


def _mix_sizes(case):
    """Vertex counts of a mix: log-uniform over a factor of 256, scaled to the case's total."""
    raw = 2.0 ** np.random.RandomState(case["graphs"]).uniform(0, 8, case["graphs"])
    return np.maximum(64, raw / raw.sum() * case["n"]).astype(np.int64)


def _mix(case, gen):
    """Half R-MAT (edge factor 8 to 32), half SBM."""
    return [_graph("rmat" if i % 2 else "sbm", int(n), (16, 32, 64)[i // 2 % 3] if i % 2 else 16, case["weighted"],
                   case["bits"], gen) for i, n in enumerate(_mix_sizes(case))]


# ---- the passes -----------------------------------------------------------------------------------

def _options(case):
    return {k: case[k] for k in ("slots", "mode") if k in case}


def _bind(graph):
    import rak_lowmem as rl
    return rl.device_csr(*graph)


def prepare(case, seed):
    import rak_lowmem as rl
    gen, kind, opts = _generator(seed), case["kind"], _options(case)
    state = {"kind": kind, "opts": opts}
    if kind != "noalloc":
        state["ctx"] = ctx = rl.Context(0)
    if kind in ("batch", "serve"):
        graphs = _mix(case, gen)
    elif kind == "set":
        graphs = [_graph(case["family"], case["n"], case["degree"], case["weighted"], case["bits"], gen)
                  for _ in range(case["graphs"])]
    else:
        graphs = [_graph(case["family"], case["n"], case["degree"], case["weighted"], case["bits"], gen)]
    torch.cuda.synchronize()
    state["graphs"] = graphs
    n = graphs[0][0].numel() - 1
    if kind == "host":
        off, tgt, wt = [None if t is None else t.cpu().numpy() for t in graphs[0]]
        state["graph"] = rl.HostGraph(off, tgt.view(np.uint32), wt)
        state["graphs"] = None
    elif kind == "noalloc":
        state["csr"], state["out"] = _bind(graphs[0]), torch.empty(n, dtype=torch.int32, device="cuda")
        state["run"] = rl.lowmem_noalloc
    elif kind == "resident":
        state["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
        state["resident"] = rl.ResidentGraph(ctx, _bind(graphs[0]), **opts)
    elif kind == "set":
        state["out"] = [torch.empty(g[0].numel() - 1, dtype=torch.int32, device="cuda") for g in graphs]
        state["resident"] = [rl.ResidentGraph(ctx, _bind(g), **opts) for g in graphs]
    elif kind == "modularity":
        # communities of 200 consecutive vertices on average, a tenth of the vertices astray
        k = max(1, n // 200)
        at = torch.arange(n, device="cuda") * k // n
        astray = torch.randint(k, (n,), device="cuda", generator=gen)
        state["labels"] = torch.where(torch.rand(n, device="cuda", generator=gen) < 0.1, astray, at).int()
        state["csr"] = _bind(graphs[0])
    elif kind == "batch":
        sizes, edges = [g[0].numel() - 1 for g in graphs], [g[1].numel() for g in graphs]
        first = np.concatenate([[0], np.cumsum(edges)])
        off = torch.cat([g[0][:-1].long() + int(e) for g, e in zip(graphs, first)] +
                        [torch.tensor([int(first[-1])], device="cuda")])
        batch = rl.DeviceBatch(torch.from_numpy(np.concatenate([[0], np.cumsum(sizes)])).cuda(), off,
                               torch.cat([g[1] for g in graphs]),
                               torch.cat([g[2] for g in graphs]) if case["weighted"] else None)
        state["graphs"], state["out"] = None, torch.empty(batch.n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        state["batch"] = rl.Batch(ctx, batch, **opts)
        state["batch"].capture(state["out"], **opts)
    elif kind == "serve":
        state["csrs"] = [_bind(g) for g in graphs]
        state["server"] = rl.Server(ctx, budget_bytes=8 << 30, max_graphs_per_launch=64, **opts)
    return state


def run(state):
    kind, opts = state["kind"], state["opts"]
    if kind == "noalloc":
        r = state["run"](0, None, state["csr"], state["out"], **opts)
        return {"membership": state["out"], "iterations": r.iterations}
    if kind == "resident":
        r = state["resident"].run(state["out"], **opts)
        return {"membership": state["out"], "iterations": r.iterations}
    if kind == "set":
        return {"modularity": np.array([g.run(m, compute_modularity=1, **opts).modularity
                                        for g, m in zip(state["resident"], state["out"])])}
    if kind == "host":
        membership, r = state["ctx"].lowmem(state["graph"], **opts)
        return {"membership": membership, "iterations": r.iterations}
    if kind == "modularity":
        return {"modularity": state["ctx"].modularity(state["csr"], state["labels"])}
    if kind == "batch":
        state["batch"].replay()
        iterations, _ = state["batch"].results()
        return {"membership": state["out"], "iterations": iterations}
    server = state["server"]
    tickets = [server.submit_device(c) for c in state["csrs"]]
    done = [server.wait(t) for t in tickets]
    return {"membership": np.concatenate([m for m, _ in done]),
            "iterations": np.array([r.iterations for _, r in done], dtype=np.int32)}


# ---- what a pass cannot do without, and what it should return -------------------------------------

def work(case):
    """Every input read once (offsets, targets, weights, and for modularity the labels), every output
    written once; one compare-and-add for each edge."""
    n, graphs = case["n"], case["graphs"] if case["kind"] == "set" else 1
    m = n * (3.8 if case["family"] == "lattice" else case["degree"] * 0.95)
    read = (n + 1) * case["bits"] // 8 + m * (8 if case["weighted"] else 4) + (4 * n if case["kind"] == "modularity" else 0)
    written = 8 if case["kind"] in ("set", "modularity") else 4 * n
    return {"bytes": graphs * (read + written), "flops": graphs * 2 * m}


def exact(case, seed):
    """Modularity in 64 bits. Memberships are whole numbers, and an asynchronous run's modularity is that of
    the communities it happens to find, so these have no exact value."""
    if case["kind"] != "modularity":
        return None
    gen = _generator(seed)
    off, tgt, wt = _graph(case["family"], case["n"], case["degree"], case["weighted"], case["bits"], gen)
    n = off.numel() - 1
    k = max(1, n // 200)
    at = torch.arange(n, device="cuda") * k // n
    astray = torch.randint(k, (n,), device="cuda", generator=gen)
    c = torch.where(torch.rand(n, device="cuda", generator=gen) < 0.1, astray, at)
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), off.long().diff())
    w = torch.ones(tgt.numel(), dtype=torch.float64, device="cuda") if wt is None else wt.double()
    total = w.sum()
    inside = w[c[src] == c[tgt.long()]].sum()
    per = torch.zeros(k, dtype=torch.float64, device="cuda").index_add_(0, c[src], w)
    return {"modularity": float(inside / total - (per * per).sum() / (total * total))}
