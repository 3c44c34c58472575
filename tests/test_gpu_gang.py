"""The single-launch stages on the GPU (one kernel per stage for batches and
levels that fit it) against the oracle, at the sizes where their shape changes:
one block, a cluster, a cooperative grid; sort chunks of 64 to 1024 records; the
largest batch they take and the first one that goes to the multi-kernel path.

Tolerance: bit-exact."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

gh = pytest.importorskip("tests.gpu_helpers")

SHAPES = {"block": (300, 900), "cluster": (20000, 90000), "grid": (60000, 420000)}
_graphs = {}


def _base(shape, integral):
    if (shape, integral) not in _graphs:
        n, m = SHAPES[shape]
        rng = np.random.default_rng(n + integral)
        s, d, w = gh.random_graph(rng, n, m, integral)
        # a hub whose row is summed apart and searched over many steps
        hub = np.setdiff1d(rng.permutation(n)[: min(n // 2, 9000)], [7]).astype(np.uint32)
        hw = np.full(len(hub), 2.0) if integral else rng.uniform(0.5, 2.0, len(hub))
        s, d = np.concatenate([s, np.full(len(hub), 7, np.uint32)]), np.concatenate([d, hub])
        g = O.Graph.from_edges(n, s, d, np.concatenate([w, hw]))
        _graphs[shape, integral] = g.apply_delta([], [], [], keep_self_loops=True)
    return _graphs[shape, integral]


def _batch(g, k, integral, seed):
    """k updates: inserts, exact deletes, weight changes, repeated keys, loops,
    many of them in the hub's row."""
    rng = np.random.default_rng(seed)
    off, col, w = g.csr()
    src = np.repeat(np.arange(g.n, dtype=np.uint32), np.diff(off).astype(np.int64))
    ds = rng.integers(0, g.n, k).astype(np.uint32)
    dd = rng.integers(0, g.n, k).astype(np.uint32)
    dw = rng.integers(-2, 4, k).astype(float) if integral else rng.uniform(-1.0, 2.5, k)
    old = rng.random(k) < 0.5
    e = rng.integers(0, len(col), k)
    ds[old], dd[old] = src[e[old]], col[e[old]]
    gone = old & (rng.random(k) < 0.6)
    dw[gone] = -w[e[gone]]
    ds[rng.random(k) < 0.2] = 7
    loop = rng.random(k) < 0.02
    dd[loop] = ds[loop]
    again = rng.random(k) < 0.1
    at = rng.integers(0, k, k)
    ds[again], dd[again] = ds[at[again]], dd[at[again]]
    return ds, dd, dw


@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("shape,k", [
    ("block", 1), ("block", 64), ("block", 65), ("block", 513),
    ("cluster", 1), ("cluster", 512), ("cluster", 1025), ("cluster", 16385),
    ("grid", 2), ("grid", 2049), ("grid", 32768), ("grid", 32769)])
def test_apply_delta_shapes(shape, k, integral):
    g = _base(shape, integral)
    for seed in range(2):
        ds, dd, dw = _batch(g, k, integral, 10 * k + seed)
        ref = g.apply_delta(ds, dd, dw, keep_self_loops=True)
        got = gh.apply_delta(g, ds, dd, dw, keep_loops=True)
        for a, b in zip(got, ref.csr()):
            assert gh.same_bits(a, b)


@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("share", [0.02, 1.0])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_inc_refinement_shapes(shape, share, integral):
    # sub-communities of 1 to a few hundred vertices inside 40 communities: rows
    # cut into slices (the hub), splits, singletons with and without candidates,
    # singletons above and below the warp table's 256 entries
    g = _base(shape, integral)
    rng = np.random.default_rng(len(shape))
    f = gh.random_partition(rng, g.n, 40)
    aff = rng.random(g.n) < share
    for subs in (3, max(4, g.n // 400), g.n // 3):
        s0 = (f.astype(np.int64) * subs + rng.integers(0, subs, g.n)) % (g.n + 5)
        s0 = np.where(rng.random(g.n) < 0.7, f * np.uint32(subs), s0).astype(np.uint32) % g.n
        for same_f in (False, True):
            ref_s, ref_r = O.inc_refinement(g, f, s0.copy(), aff, 1.0, O.MODE_THROUGHPUT,
                                            cc_same_community=same_f)
            got_s, got_r = gh.inc_refinement(g, f, s0, aff, 1.0, same_f)
            assert np.array_equal(ref_s, got_s) and np.array_equal(ref_r, got_r)


# 40000 updates: the batch, and more than 65536 aggregation records, take the
# multi-kernel path on the lower levels
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("shape,ks", [("block", (1, 40, 400)), ("cluster", (3, 700, 9000)),
                                      ("grid", (50, 5000, 40000))])
def test_levels_match_oracle(shape, ks, integral):
    from tests.test_gpu_e2e import compare, oracle_state

    import importlib
    hl = importlib.import_module("hit-leiden_b200")
    g = _base(shape, integral)
    off, col, w = g.csr()
    src = np.repeat(np.arange(g.n, dtype=np.uint32), np.diff(off).astype(np.int64))
    once = src < col
    edges = src[once], col[once], w[once]
    gs = hl.PartitionState.load(hl.GraphInput.from_arrays(shape, g.n, *edges),
                                hl.RunConfig(mode=hl.RunMode.Throughput))
    ref = oracle_state(g.n, *edges, 10)
    compare(gs, ref)
    for i, k in enumerate(ks):
        ds, dd, dw = _batch(g, k, integral, 77 + i)
        gs.apply_batch(ds, dd, dw)
        ref.hit_leiden(ds, dd, dw)
        compare(gs, ref)
    gs.close()


@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("labels", ["few", "many", "high"])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_inc_movement_shapes(shape, labels, integral):
    # few: the hub's row holds 40 keys, long chains; many: more than 2048 keys,
    # so the round goes to the multi-kernel path; high: ids of n and above are
    # compacted first.  From a batch, and from all vertices (60,000 of them
    # outgrow the frontier lists).
    g = _base(shape, integral)
    rng = np.random.default_rng(len(labels))
    f = gh.random_partition(rng, g.n, 40 if labels == "few" else g.n // 2)
    if labels == "high":
        f = (f + np.uint32(g.n // 2 + 3)).astype(np.uint32)
    s = gh.random_partition(rng, g.n, g.n // 3)
    for k in (0, min(2000, g.n // 4)):
        ds, dd, dw = _batch(g, k, integral, 5) if k else ([], [], [])
        for rounds in ((1, 20) if shape == "block" else (2,)):
            ref = O.inc_movement(g, ds, dd, dw, f.copy(), s, 1.0, O.MODE_THROUGHPUT,
                                 max_rounds=rounds)
            got = gh.inc_movement(g, ds, dd, dw, f, s, 1.0, max_rounds=rounds)
            assert np.array_equal(ref[0], got[0])
            assert np.array_equal(ref[1], got[1]) and np.array_equal(ref[2], got[2])


# Rows above 64 entries carry bounds from round to round (prune.cuh): dense
# graphs with few communities keep whole neighbourhoods active for 20 rounds,
# in the one-launch and in the multi-kernel rounds.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("gamma", [0.0, 0.7, 3.0])
@pytest.mark.parametrize("multi", [False, True])
def test_bounds_change_nothing(integral, gamma, multi):
    import importlib
    hl = importlib.import_module("hit-leiden_b200")
    rng = np.random.default_rng(int(10 * gamma) + integral)
    n = 1500
    s, d, w = gh.random_graph(rng, n, 90000, integral)
    cfg = hl.RunConfig(mode=hl.RunMode.Throughput, resolution=gamma, small_rounds=not multi)
    gs = hl.PartitionState.load(hl.GraphInput.from_arrays("dense", n, s, d, w), cfg)
    ref = O.State(n, gamma=gamma, mode=O.MODE_THROUGHPUT)
    ref.bootstrap(s, d, w, max_levels=10)
    for i in range(3):
        ds = rng.integers(0, n, 400).astype(np.uint32)
        dd = rng.integers(0, n, 400).astype(np.uint32)
        dw = rng.integers(1, 9, 400).astype(float) if integral else rng.uniform(0.1, 9.0, 400)
        gs.apply_batch(ds, dd, dw)
        ref.hit_leiden(ds, dd, dw)
        assert gs.levels == ref.levels
        for p in range(ref.levels):
            assert np.array_equal(gs.community_mapping_per_level[p], ref.get_map(p, O.MAP_F))
            assert np.array_equal(gs.current_subcommunity_mapping_per_level[p],
                                  ref.get_map(p, O.MAP_S_CUR))
    gs.close()


# Deterministic mode takes up to 128 pops together and keeps its state in shared
# memory by size: bit sets, labels (32768 nodes) and community degrees (10240).
# Rows above 128 entries take the whole block.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("n,m", [(60, 200), (10240, 21000), (10241, 21000), (33000, 60000)])
def test_deterministic_sizes(n, m, integral):
    import importlib
    hl = importlib.import_module("hit-leiden_b200")
    rng = np.random.default_rng(n)
    s, d, w = gh.random_graph(rng, n, m, integral)
    hub = rng.permutation(n)[: min(n // 2, 700)].astype(np.uint32)
    hub = hub[hub != 3]
    s, d = np.concatenate([s, np.full(len(hub), 3, np.uint32)]), np.concatenate([d, hub])
    w = np.concatenate([w, np.ones(len(hub)) if integral else rng.uniform(0.5, 2.0, len(hub))])
    gs = hl.PartitionState.load(hl.GraphInput.from_arrays("det", n, s, d, w),
                                hl.RunConfig(mode=hl.RunMode.Deterministic, max_iterations=1))
    ref = O.State(n, levels=1, mode=O.MODE_DETERMINISTIC)
    ref.push_empty_graph()
    ref.hit_leiden(s, d, w)
    for i in range(2):
        ds = rng.integers(0, n, 200).astype(np.uint32)
        dd = rng.integers(0, n, 200).astype(np.uint32)
        dw = rng.integers(1, 4, 200).astype(float) if integral else rng.uniform(0.5, 2.0, 200)
        gs.apply_batch(ds, dd, dw)
        ref.hit_leiden(ds, dd, dw)
        assert np.array_equal(gs.community_mapping_per_level[0], ref.get_map(0, O.MAP_F))
        assert np.array_equal(gs.current_subcommunity_mapping_per_level[0],
                              ref.get_map(0, O.MAP_S_CUR))
    gs.close()


@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_modularity_and_partition_shapes(shape, integral):
    # labels: one community, a few large ones, one vertex each, values far above
    # n; the hub's row and long communities take a whole warp
    import importlib
    hl = importlib.import_module("hit-leiden_b200")
    g = _base(shape, integral)
    off, col, w = g.csr()
    src = np.repeat(np.arange(g.n, dtype=np.uint32), np.diff(off).astype(np.int64))
    once = src < col
    st = hl.PartitionState.load(
        hl.GraphInput.from_arrays(shape, g.n, src[once], col[once], w[once]),
        hl.RunConfig(mode=hl.RunMode.Throughput, max_iterations=1))
    ref = O.Graph.from_edges(g.n, src[once], col[once], w[once])
    rng = np.random.default_rng(3)
    for part in (np.zeros(g.n, np.uint32), rng.integers(0, 5, g.n).astype(np.uint32),
                 np.arange(g.n, dtype=np.uint32),
                 (rng.integers(0, 300, g.n) * 70001).astype(np.uint32)):
        q = O.modularity_csr(ref, part)
        assert abs(st.modularity(part) - q) <= 1e-12 * max(1.0, abs(q))
    assert np.array_equal(st.partition(), O.canonicalize(st.community_mapping_per_level[0]))
    st.close()


# From 148 rows above 512 entries and 65,536 others on, the two kinds are
# evaluated on two streams; one hub or one vertex fewer keeps a single one.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("hubs,others", [(148, 65536), (147, 65536), (148, 65535)])
def test_hub_rows_beside_the_others(hubs, others, integral):
    n = hubs + others
    rng = np.random.default_rng(n + integral)
    s = np.concatenate([np.repeat(np.arange(hubs), 700), rng.integers(hubs, n, 2 * n),
                        np.arange(hubs, n)])
    d = np.concatenate([rng.integers(hubs, n, 700 * hubs), rng.integers(hubs, n, 2 * n),
                        np.roll(np.arange(hubs, n), 1)])
    w = np.ones(len(s)) if integral else rng.uniform(0.5, 2.0, len(s))
    g = O.Graph.from_edges(n, s.astype(np.uint32), d.astype(np.uint32), w)
    f = gh.random_partition(rng, n, n // 20)
    sub = np.arange(n, dtype=np.uint32)
    ref = O.inc_movement(g, [], [], [], f.copy(), sub, 1.0, O.MODE_THROUGHPUT, max_rounds=3)
    got = gh.inc_movement(g, [], [], [], f, sub, 1.0, max_rounds=3)
    assert all(np.array_equal(ref[i], got[i]) for i in range(3))
