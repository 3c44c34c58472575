"""The work that programs give this library, as timed cases.

A program holds graphs resident on the GPU, feeds them batches of edge updates
and reads the hierarchical partition back.  The listed cases go from a handful
of updates on a few hundred vertices to the large graphs of the benchmark
configurations (LFR-style f64 weights with 1M vertices; R-MAT with unit
weights), through both run modes, one level and many, the many-graph form, a
load from scratch and the modularity of a given partition.  ``draw`` gives more
cases of the same kinds with sizes spread over the same ranges.

A pass over a resident graph applies a batch, reads the partition, applies the
batch that undoes it and reads the partition again, as a program with a sliding
window of edges does: the graph is the same at the start of every pass, so a
state can be updated any number of times.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

hl = importlib.import_module("hit-leiden_b200")
workloads = importlib.import_module("hit-leiden_b200.workloads")


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _update(graph, n, degree, weights, updates, inserts, mode="throughput", levels=10,
            resolution=1.0, mu=0.25, **more):
    return dict(kind="update", graph=graph, n=n, degree=degree, weights=weights, updates=updates,
                inserts=inserts, mode=mode, levels=levels, resolution=resolution, mu=mu, **more)


def listed():
    return [
        # a small social graph that follows single events: latency of one call
        dict(name="tiny_stream", **_update("planted", 403, 6.0, "unit", 16, 0.8)),
        # the collaboration graph of the small benchmark configuration
        # (9,877 vertices, mean degree 4.4, 1,000 new edges a batch)
        dict(name="collab_batch", **_update("planted", 9877, 4.4, "unit", 1000, 1.0, mu=0.15)),
        # the same graph in the default, deterministic mode
        dict(name="collab_default", **_update("planted", 9877, 4.4, "unit", 1000, 1.0, mu=0.15,
                                              mode="deterministic")),
        # the single-level state of the reference crate, real weights, a finer
        # resolution
        dict(name="one_level", **_update("planted", 99991, 16.0, "real", 5000, 0.5, levels=1,
                                         resolution=1.5)),
        # a mid-size community graph, 2% of its edges changed
        dict(name="community_50k", **_update("planted", 50021, 12.0, "unit", 6000, 0.8)),
        # LFR-style graph, f64 weights, 10k updates (90% inserts): the mid-size
        # benchmark configuration
        dict(name="weighted_1m", **_update("planted", 1000000, 40.0, "real", 10000, 0.9, mu=0.3)),
        # R-MAT graphs, unit weights, hubs of many thousand neighbours: the
        # large benchmark configuration at two smaller scales
        dict(name="rmat_17", **_update("rmat", 1 << 17, 32.0, "unit", 3906, 0.9)),
        dict(name="rmat_21", **_update("rmat", 1 << 21, 32.0, "unit", 62500, 0.9)),
        # many graphs of uneven size, each with its own batch (1-5% of its edges)
        dict(name="many_graphs", kind="many", graphs=48, n_lo=1000, n_hi=30000, weights="unit",
             workers=16),
        # load a graph from scratch and take its partition and modularity
        dict(name="load_small", kind="load", graph="planted", n=9877, degree=4.4, weights="unit",
             mu=0.15, mode="throughput"),
        dict(name="load_300k", kind="load", graph="planted", n=300007, degree=20.0,
             weights="real", mu=0.25, mode="throughput"),
        # quality of a partition from elsewhere on a resident graph
        dict(name="modularity_500k", kind="quality", n=500009, degree=24.0, weights="real",
             mu=0.25, parts=4000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["planted", "planted", "planted", "default", "one_level", "rmat", "many",
                       "load", "quality"])
    weights = rng.choice(["unit", "unit", "real", "counts"])
    degree = round(rng.uniform(4.0, 40.0), 1)
    mu = round(rng.uniform(0.1, 0.4), 2)
    inserts = rng.choice([0.0, 0.5, 0.8, 0.9, 1.0])
    if kind == "rmat":
        n = 1 << rng.randint(14, 20)
        return _update("rmat", n, 32.0, "unit", _log_uniform(rng, 100, n // 32 + 100), inserts)
    if kind == "many":
        lo = _log_uniform(rng, 300, 3000)
        return dict(kind="many", graphs=rng.randint(4, 60), n_lo=lo, n_hi=lo * rng.randint(2, 20),
                    weights=weights, workers=rng.choice([4, 8, 16]))
    if kind == "load":
        return dict(kind="load", graph="planted", n=_log_uniform(rng, 300, 300000), degree=degree,
                    weights=weights, mu=mu, mode="throughput")
    if kind == "quality":
        n = _log_uniform(rng, 1000, 800000)
        return dict(kind="quality", n=n, degree=degree, weights=weights, mu=mu,
                    parts=_log_uniform(rng, 2, max(3, n // 10)))
    if kind == "default":
        n = _log_uniform(rng, 300, 10000)
        return _update("planted", n, round(rng.uniform(3.0, 8.0), 1), weights,
                       _log_uniform(rng, 4, max(8, n // 10)), inserts, mode="deterministic", mu=mu)
    n = _log_uniform(rng, 300, 700000)
    updates = _log_uniform(rng, 4, max(16, min(20000, int(n * degree * 0.02))))
    return _update("planted", n, degree, weights, updates, inserts,
                   levels=1 if kind == "one_level" else 10,
                   resolution=rng.choice([0.5, 1.0, 1.0, 2.0]), mu=mu)


# ---------------------------------------------------------------------------
# Seeded graphs and batches, generated on the GPU
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weights(kind, m, gen):
    if kind == "unit":
        return torch.ones(m, dtype=torch.float64, device="cuda")
    r = torch.rand(m, generator=gen, dtype=torch.float64, device="cuda")
    return 0.5 + 1.5 * r if kind == "real" else torch.floor(1.0 + 9.0 * r)


def _planted(n, degree, mu, weights, seed):
    """Power-law degrees (exponent 2.5) and community sizes (exponent 1.5), a
    share mu of every vertex's edges outside its community."""
    gen = _generator(seed)
    rnd = lambda k: torch.rand(k, generator=gen, dtype=torch.float64, device="cuda")  # noqa: E731
    top = max(8.0, min(2000.0, 4.0 * math.sqrt(n)))
    # a little above the wanted mean: duplicate pairs and loops fall away
    deg = torch.clamp(degree * 1.1 / 3.0 * (1.0 - rnd(n)) ** (-1.0 / 1.5), 1.0, top)
    deg = torch.floor(deg + rnd(n)).to(torch.int64)
    lo, hi = max(3.0, min(50.0, n / 40.0)), max(6.0, min(5000.0, n / 8.0))
    q = rnd(int(n / lo) + 1)
    sizes = (lo ** -0.5 + q * (hi ** -0.5 - lo ** -0.5)) ** -2.0
    ends = torch.cumsum(torch.ceil(sizes), 0)
    place = torch.argsort(rnd(n)).to(torch.float64)
    comm = torch.searchsorted(ends, place, right=True)
    inside = torch.floor(deg * (1.0 - mu) + rnd(n)).to(torch.int64).clamp(max=deg)
    ids = torch.arange(n, device="cuda")
    stub = torch.repeat_interleave(ids, inside)
    stub = stub[torch.argsort(comm[stub].to(torch.float64) + rnd(stub.numel()))]
    stub = stub[: stub.numel() // 2 * 2].view(-1, 2)
    stub = stub[comm[stub[:, 0]] == comm[stub[:, 1]]]
    far = torch.repeat_interleave(ids, deg - inside)
    far = far[torch.argsort(rnd(far.numel()))]
    far = far[: far.numel() // 2 * 2].view(-1, 2)
    pairs = torch.cat([stub, far])
    a, b = pairs.min(1).values, pairs.max(1).values
    key = torch.unique((a * n + b)[a != b])
    return key // n, key % n, _weights(weights, key.numel(), gen)


def _graph(case, seed):
    if case["graph"] == "rmat":
        n, src, dst = workloads.rmat_torch(int(math.log2(case["n"])), int(case["degree"] // 2),
                                           seed)
        return src, dst, torch.ones(src.numel(), dtype=torch.float64, device="cuda")
    return _planted(case["n"], case["degree"], case["mu"], case["weights"], seed)


def _host(u, v, w=None):
    u, v = u.to(torch.int32).cpu().numpy().view(np.uint32), v.to(torch.int32).cpu().numpy()
    return u, v.view(np.uint32), None if w is None else w.cpu().numpy()


def _batch(case, n, src, dst, w, updates, inserts, seed):
    """One batch: new pairs (end points drawn by degree, as a random end of a
    random edge; R-MAT pairs on R-MAT graphs) and deletes of distinct edges."""
    gen = _generator(seed)
    m = src.numel()
    ki = int(round(updates * inserts))
    kd = min(updates - ki, m // 4)
    if case.get("graph") == "rmat":
        u, v, _ = workloads.rmat_batch_torch(int(math.log2(n)), src, dst, ki, 1.0, seed)
        u, v = u.long(), v.long()
    else:
        e = torch.randint(0, m, (2, ki), generator=gen, device="cuda")
        u, v = src[e[0]].long(), dst[e[1]].long()
        v = torch.where(u == v, (v + 1) % n, v)
    d = torch.unique(torch.randint(0, m, (kd,), generator=gen, device="cuda"))
    u, v = torch.cat([u, src[d].long()]), torch.cat([v, dst[d].long()])
    dw = torch.cat([_weights(case["weights"], ki, gen), -w[d]])
    mix = torch.randperm(u.numel(), generator=gen, device="cuda")
    return u[mix], v[mix], dw[mix]


def _batches(case, n, src, dst, w, updates, inserts, seed):
    u, v, dw = _batch(case, n, src, dst, w, updates, inserts, seed * 1000003 + 7)
    return [_host(u, v, dw), _host(u, v, -dw)]


def _config(case):
    mode = hl.RunMode.Deterministic if case["mode"] == "deterministic" else hl.RunMode.Throughput
    return hl.RunConfig(mode=mode, resolution=case.get("resolution", 1.0),
                        max_iterations=case.get("levels", 10))


# ---------------------------------------------------------------------------
# Preparing and running a case
# ---------------------------------------------------------------------------
def _many_sizes(case, seed):
    r = np.random.default_rng(seed)
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    # evenly spread over the logarithm, so that every seed has the same work
    at = (np.arange(case["graphs"]) + 0.5) / case["graphs"]
    sizes = np.exp(lo + at * (hi - lo)).astype(int)
    return [(int(n), float(r.uniform(4.0, 32.0)), float(r.uniform(0.1, 0.4)),
             float(r.uniform(0.01, 0.05))) for n in sizes]


def prepare(case, seed):
    if case["kind"] == "many":
        states, batches = [], []
        cfg = hl.RunConfig(mode=hl.RunMode.Throughput)
        for i, (n, degree, mu, share) in enumerate(_many_sizes(case, seed)):
            src, dst, w = _planted(n, degree, mu, case["weights"], seed * 4099 + i)
            states.append(hl.PartitionState.load(
                hl.GraphInput.from_arrays(f"g{i}", n, *_host(src, dst, w)), cfg))
            batches.append(_batches(case, n, src, dst, w, max(4, int(share * src.numel())), 0.8,
                                    seed * 4099 + i))
        return dict(kind="many", states=states, batches=batches, workers=case["workers"])
    if case["kind"] == "load":
        src, dst, w = _graph(case, seed)
        g = hl.GraphInput.from_arrays("load", case["n"], *_host(src, dst, w))
        return dict(kind="load", graph=g, config=_config(case))
    if case["kind"] == "quality":
        n = case["n"]
        src, dst, w = _planted(n, case["degree"], case["mu"], case["weights"], seed)
        state = hl.PartitionState.load(
            hl.GraphInput.from_arrays("quality", n, *_host(src, dst, w)),
            hl.RunConfig(mode=hl.RunMode.Throughput, max_iterations=1))
        return dict(kind="quality", state=state, part=_parts(case, seed))
    src, dst, w = _graph(case, seed)
    n = case["n"]
    state = hl.PartitionState.load(hl.GraphInput.from_arrays("update", n, *_host(src, dst, w)),
                                   _config(case))
    return dict(kind="update", state=state,
                batches=_batches(case, n, src, dst, w, case["updates"], case["inserts"], seed))


def _parts(case, seed):
    """A partition with communities of uneven size."""
    r = np.random.default_rng(seed + 17)
    return (r.random(case["n"]) ** 2 * case["parts"]).astype(np.uint32)


def run(state):
    if state["kind"] == "load":
        out = hl.run(state["graph"], state["config"]).partition
        return [out.node_to_community, out.quality_score]
    if state["kind"] == "quality":
        return state["state"].modularity(state["part"])
    out = []
    for turn in range(2):
        if state["kind"] == "many":
            states = state["states"]
            hl.apply_batches(states, [b[turn] for b in state["batches"]],
                             workers=state["workers"])
            out.append(np.concatenate([s.partition() for s in states]))
        else:
            s = state["state"]
            s.apply_batch(*state["batches"][turn])
            out += [s.partition(), s.node_to_comm]
    return out


# ---------------------------------------------------------------------------
# Work and exact values
# ---------------------------------------------------------------------------
def work(case):
    """Bytes no pass can do without.  Adjacency entries hold a neighbour (4) and
    a weight (8); reading one for a decision also takes its neighbour's label."""
    if case["kind"] == "many":
        total = 0
        for n, degree, _, share in _many_sizes(case, 0):
            k = share * n * degree / 2
            total += 2 * (16 * k + 2 * k * degree * 16 + 4 * n)
        return {"bytes": total}
    n, degree = case["n"], case["degree"]
    entries = n * degree
    if case["kind"] == "load":  # edges in, both directions stored and read once
        return {"bytes": 8 * entries + 12 * entries + 16 * entries + 8 * n}
    if case["kind"] == "quality":
        return {"bytes": 16 * entries + 12 * n, "flops": entries + 2 * n}
    # two batches: the edges, the rows of their end points, two label maps out
    k = case["updates"]
    return {"bytes": 2 * (16 * k + 2 * k * degree * 16 + 8 * n)}


def _modularity(n, u, v, w, part):
    """Modularity of a partition, term by term in 64 bits."""
    two_m = 2.0 * math.fsum(w)
    deg = np.bincount(u, weights=w, minlength=n) + np.bincount(v, weights=w, minlength=n)
    inside = 2.0 * math.fsum(w[part[u] == part[v]])
    tot = np.bincount(part, weights=deg)
    return inside / two_m - math.fsum((tot / two_m) ** 2)


def exact(case, seed):
    if case["kind"] == "quality":
        u, v, w = _host(*_planted(case["n"], case["degree"], case["mu"], case["weights"], seed))
        return _modularity(case["n"], u.astype(np.int64), v.astype(np.int64), w,
                           _parts(case, seed).astype(np.int64))
    # partitions are whole numbers; the loaded state's modularity follows from
    # its own partition, which only the library computes
    return None
