"""The update path at the limits of its counters, lists and scratch, on the GPU
against the oracle.

Tolerance: bit-exact."""
import importlib

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

gh = pytest.importorskip("tests.gpu_helpers")
hl = importlib.import_module("hit-leiden_b200")
W = importlib.import_module("hit-leiden_b200.workloads")


def _load(n, edges, **config):
    return hl.PartitionState.load(hl.GraphInput.from_arrays("limits", n, *edges),
                                  hl.RunConfig(mode=hl.RunMode.Throughput, **config))


def _oracle(n, edges, max_levels=10, **more):
    ref = O.State(n, mode=O.MODE_THROUGHPUT, **more)
    ref.bootstrap(*edges, max_levels=max_levels)
    return ref


def _same(gs, ref):
    assert gs.levels == ref.levels
    for p in range(ref.levels):
        assert np.array_equal(gs.community_mapping_per_level[p], ref.get_map(p, O.MAP_F))
        assert np.array_equal(gs.current_subcommunity_mapping_per_level[p],
                              ref.get_map(p, O.MAP_S_CUR))


def _updates(rng, n, edges, k, integral):
    """New random edges and exact deletes, half of each."""
    s, d, w = edges
    e = rng.choice(len(s), k, replace=False)
    u = np.concatenate([rng.integers(0, n, k).astype(np.uint32), s[e]])
    v = np.concatenate([rng.integers(0, n, k).astype(np.uint32), d[e]])
    new = rng.integers(1, 4, k).astype(float) if integral else rng.uniform(0.5, 2.0, k)
    return u, v, np.concatenate([new, -w[e]])


def _double_star(leaves, integral):
    """Two hubs joined by an edge.  After the load the leaves of a hub are one
    sub-community without the hub, which any edge inside it splits to pieces."""
    at = np.arange(leaves, dtype=np.uint32)
    s = np.concatenate([np.zeros(leaves), np.ones(leaves), [0]]).astype(np.uint32)
    d = np.concatenate([at + 2, at + leaves + 2, [1]]).astype(np.uint32)
    rng = np.random.default_rng(leaves)
    return 2 * leaves + 2, (s, d, np.ones(len(s)) if integral else rng.uniform(0.5, 2.0, len(s)))


# One inserted edge changes the rows of all leaves: fewer aggregation records
# than the one-launch form takes, more records, more changed rows.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("leaves", [30000, 40000, 66000, 90000])
def test_one_edge_changes_many_rows(leaves, integral):
    n, edges = _double_star(leaves, integral)
    gs, ref = _load(n, edges), _oracle(n, edges)
    before = ref.get_map(0, O.MAP_S_CUR)
    for u, v in ((2, 3), (leaves + 2, leaves + 3)):
        b = np.array([u], np.uint32), np.array([v], np.uint32), np.ones(1)
        gs.apply_batch(*b)
        ref.hit_leiden(*b)
        _same(gs, ref)
    if integral:
        assert np.sum(before != ref.get_map(0, O.MAP_S_CUR)) > 2 * leaves - 10
    gs.close()


# The records that outgrow the one launch are counted, not sorted: its share of
# a batch that changes a million rows stays below a few milliseconds (27 ms when
# the changed rows were sorted first).
def test_changed_rows_are_not_sorted_in_vain():
    n, edges = _double_star(1000000, True)
    gs = _load(n, edges, kernel_timing=True)
    gs.apply_batch(np.array([2], np.uint32), np.array([3], np.uint32), np.ones(1))
    ms = gs.kernel_stats()["aggregate_one_launch"]["ms"]
    gs.close()
    assert ms < 5.0, ms


# Two million vertices in two communities: their integral degrees add up in the
# warp before they meet on one word (3.1 ms for this batch's two levels without).
def test_degrees_of_giant_communities():
    n, edges = _double_star(1000000, True)
    gs = _load(n, edges, kernel_timing=True)
    ref = _oracle(n, edges)
    for i in range(2):
        before = gs.kernel_stats()["move_one_launch"]["ms"]
        b = np.array([2 + i], np.uint32), np.array([40 + i], np.uint32), np.ones(1)
        gs.apply_batch(*b)
        ref.hit_leiden(*b)
        _same(gs, ref)
        ms = gs.kernel_stats()["move_one_launch"]["ms"] - before
        assert ms < 1.5, ms
    gs.close()


# Eight thousand vertices change community in one round, f64 weights: d(C) of
# the two communities takes their degrees in selected order, by a warp each (2.8
# ms of movement by a thread each, 0.9 so).
def test_thousands_of_moves_into_one_community():
    leaves = 8000
    n, edges = _double_star(leaves, False)
    gs, ref = _load(n, edges, kernel_timing=True), _oracle(n, edges)
    at = np.arange(2, leaves + 2, dtype=np.uint32)
    best = 1e9
    for i in range(4):
        for w in (5.25, -5.25):
            b = np.ones(leaves, np.uint32), at, np.full(leaves, w)
            before = gs.kernel_stats()["move_one_launch"]["ms"]
            moved = gs.apply_batch(*b).moves
            ms = gs.kernel_stats()["move_one_launch"]["ms"] - before
            if w > 0.0:
                assert moved > leaves
                best = min(best, ms)
            ref.hit_leiden(*b)
            _same(gs, ref)
    assert best < 1.8, best
    gs.close()


# Rows at and above the 16,384 entries the hub tables take: a longer one hands
# the round back before it is evaluated, from a batch that touches it, from one
# that makes its neighbours move, and where its bound rules it out.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("deg", [16384, 16385, 30000])
def test_hub_longer_than_its_tables(deg, integral):
    rng = np.random.default_rng(deg)
    n = 40000
    s, d, w = gh.random_graph(rng, n, 120000, integral)
    hub = rng.choice(np.arange(1, n, dtype=np.uint32), deg, replace=False)
    keep = s != 0
    keep &= d != 0
    s, d, w = s[keep], d[keep], w[keep]
    s = np.concatenate([s, np.zeros(deg, np.uint32)])
    d = np.concatenate([d, hub])
    w = np.concatenate([w, np.ones(deg) if integral else rng.uniform(0.5, 2.0, deg)])
    gs, ref = _load(n, (s, d, w)), _oracle(n, (s, d, w))
    _same(gs, ref)
    for i in range(3):
        k = (10, 3000, 9000)[i]
        u = rng.integers(0, n, k).astype(np.uint32)
        v = rng.integers(0, n, k).astype(np.uint32)
        if i == 0:
            u[:5] = 0
        b = u, v, np.full(k, 3.0) if integral else rng.uniform(2.0, 4.0, k)
        gs.apply_batch(*b)
        ref.hit_leiden(*b)
        _same(gs, ref)
    gs.close()


def _same_det(gs, ref):
    assert np.array_equal(gs.community_mapping_per_level[0], ref.get_map(0, O.MAP_F))
    assert np.array_equal(gs.current_subcommunity_mapping_per_level[0],
                          ref.get_map(0, O.MAP_S_CUR))


def _load_det(n, edges, gamma=1.0, **config):
    gs = hl.PartitionState.load(
        hl.GraphInput.from_arrays("det", n, *edges),
        hl.RunConfig(mode=hl.RunMode.Deterministic, max_iterations=1, resolution=gamma, **config))
    ref = O.State(n, levels=1, mode=O.MODE_DETERMINISTIC, gamma=gamma)
    ref.push_empty_graph()
    ref.hit_leiden(*edges)
    return gs, ref


# Deterministic mode where every other row is above the 128 entries a warp
# takes: lists that end at a long row at any place, keys shared by many of a
# row's entries and by none.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("gamma", [0.2, 1.0, 4.0])
def test_deterministic_long_rows(integral, gamma):
    rng = np.random.default_rng(17)
    n = 900
    s = (n * rng.random(60000) ** 3).astype(np.uint32)
    d = (n * rng.random(60000) ** 1.5).astype(np.uint32)
    s, d = s[s != d], d[s != d]
    w = np.ones(len(s)) if integral else rng.uniform(0.5, 2.0, len(s))
    gs, ref = _load_det(n, (s, d, w), gamma)
    _same_det(gs, ref)
    for k in (1, 30, 300):
        u, v = rng.integers(0, n, k).astype(np.uint32), rng.integers(0, n, k).astype(np.uint32)
        b = u, v, np.full(k, 40.0) if integral else rng.uniform(10.0, 60.0, k)
        gs.apply_batch(*b)
        ref.hit_leiden(*b)
        _same_det(gs, ref)
    gs.close()


# A singleton with a short row beside sub-communities on both sides of the size
# from which the block sums w(S, C); the sum is kept while members join.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("leaves", [500, 2047, 2048, 3000])
def test_deterministic_merges_beside_large_subcommunities(leaves, integral):
    n, edges = _double_star(leaves, integral)
    gs, ref = _load_det(n, edges)
    _same_det(gs, ref)
    for i in range(3):
        at = slice(i * 20, i * 20 + 1 + 9 * i)
        cut = edges[0][at], edges[1][at], -edges[2][at]
        for b in (cut, (cut[0], cut[1], -cut[2])):
            gs.apply_batch(*b)
            ref.hit_leiden(*b)
            _same_det(gs, ref)
    gs.close()


# The walk's time on a graph of hubs (R-MAT 2^17): 4.8 to 6.2 ms of movement a
# pass while rows beyond a long one were evaluated in vain, 2.5 so.
def test_deterministic_hub_rows_time():
    scale = 17
    n, s, d = W.rmat_torch(scale, 16, 3)
    u, v, _ = W.rmat_batch_torch(scale, s, d, 80, 1.0, 5)
    s, d, u, v = (x.cpu().numpy().astype(np.uint32) for x in (s, d, u, v))
    gs = hl.PartitionState.load(
        hl.GraphInput.from_arrays("det", n, s, d, np.ones(len(s))),
        hl.RunConfig(mode=hl.RunMode.Deterministic, resolution=0.2, kernel_timing=True))
    best = 1e9
    for _ in range(5):
        before = gs.kernel_stats()["stage_move"]["ms"]
        gs.apply_batch(u, v, np.ones(len(u)))
        gs.apply_batch(u, v, -np.ones(len(u)))
        best = min(best, gs.kernel_stats()["stage_move"]["ms"] - before)
    gs.close()
    assert best < 4.4, best


def _hubs(n, m, integral, hubs):
    rng = np.random.default_rng(5)
    s, d = rng.integers(0, n, m), rng.integers(0, n, m)
    for h in range(hubs):
        s = np.concatenate([s, np.full(n // 4, h)])
        d = np.concatenate([d, rng.choice(n, n // 4, replace=False)])
    s, d = s[s != d].astype(np.uint32), d[s != d].astype(np.uint32)
    return s, d, rng.integers(1, 4, len(s)).astype(float) if integral else rng.uniform(0.5, 2.0,
                                                                                       len(s))


# Budgets that just hold a load, two batches, their partitions and modularities
# by the multi-kernel stages: the one-launch stages and the bounds take more, and
# a handle that cannot hold that does without them.  Results as without a budget.
@pytest.mark.parametrize("n,m,integral,hubs,mode,levels,budget", [
    (20000, 80000, True, 0, "Throughput", 10, 28131662),
    (20000, 80000, False, 0, "Throughput", 10, 33116190),
    (20000, 60000, True, 6, "Throughput", 10, 31103129),
    (20000, 60000, False, 6, "Throughput", 10, 163400974),
    (50000, 100000, False, 0, "Throughput", 1, 33567747),
    (3000, 9000, True, 0, "Deterministic", 10, 3903253),
    (3000, 9000, False, 0, "Deterministic", 10, 5542577)])
def test_tight_budgets(n, m, integral, hubs, mode, levels, budget):
    edges = _hubs(n, m, integral, hubs)
    rng = np.random.default_rng(6)
    batches = [_updates(rng, n, edges, k, integral) for k in (50, 2000)]
    out = []
    for b in (budget, 0):
        gs = hl.PartitionState.load(
            hl.GraphInput.from_arrays("budget", n, *edges),
            hl.RunConfig(mode=hl.RunMode[mode], max_iterations=levels, hbm_budget=b))
        out.append([])
        for u, v, w in batches:
            gs.apply_batch(u, v, w)
            out[-1] += [gs.partition(), gs.modularity(), *gs.community_mapping_per_level,
                        *gs.current_subcommunity_mapping_per_level]
        gs.close()
    assert len(out[0]) == len(out[1])
    for a, b in zip(*out):
        if isinstance(a, float):
            assert abs(a - b) <= 1e-12 * max(1.0, abs(b))
        else:
            assert np.array_equal(a, b)


# A generous budget keeps the one-launch stages.  Its CSR buffers have no room up
# front, so the delta goes in two launches that share one counter block: the size
# first, then the rest.  Weight changes only, then structure, several times over.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("mode", ["Throughput", "Deterministic"])
def test_generous_budget(integral, mode):
    n = 4000
    edges = _hubs(n, 12000, integral, 2)
    key = np.unique(np.minimum(edges[0], edges[1]).astype(np.int64) * n
                    + np.maximum(edges[0], edges[1]))
    edges = ((key // n).astype(np.uint32), (key % n).astype(np.uint32), edges[2][:len(key)])
    cfg = hl.RunConfig(mode=hl.RunMode[mode], max_iterations=1, hbm_budget=8 << 30,
                       kernel_timing=True)
    gs = hl.PartitionState.load(hl.GraphInput.from_arrays("budget", n, *edges), cfg)
    ref = O.State(n, levels=1,
                  mode=O.MODE_THROUGHPUT if mode == "Throughput" else O.MODE_DETERMINISTIC)
    ref.push_empty_graph()
    ref.hit_leiden(*edges)
    rng = np.random.default_rng(9)
    e = rng.choice(len(edges[0]), 300, replace=False)
    more = np.ones(300) if integral else rng.uniform(0.5, 1.0, 300)
    weights = edges[0][e], edges[1][e], more  # existing edges only
    for i in range(8):
        b = weights if i in (0, 1, 4) else _updates(rng, n, edges, (1, 40, 600)[i % 3], integral)
        before = gs.kernel_stats()["apply_one_launch"]["launches"]
        gs.apply_batch(*b)
        assert gs.kernel_stats()["apply_one_launch"]["launches"] > before
        ref.hit_leiden(*b)
        _same_det(gs, ref)
        off, col, wt = gs.supergraph(0)
        ro, rc, rw = ref.graph(0).csr()
        assert np.array_equal(off, ro) and np.array_equal(col, rc) and gh.same_bits(wt, rw)
    gs.close()


# A level of more entries than the second buffer gets room for up front: the
# same two launches, without a budget.
def test_delta_of_a_large_level_in_two_launches():
    rng = np.random.default_rng(2)
    n, m = 400000, 2200000
    s, d, w = gh.random_graph(rng, n, m, False)
    g = O.Graph.from_edges(n, s, d, w).apply_delta([], [], [], keep_self_loops=True)
    off, col, _ = g.csr()
    assert len(col) > 1 << 22
    for k in (1, 3000):
        e = rng.integers(0, len(s), k)
        u = np.concatenate([rng.integers(0, n, k).astype(np.uint32), s[e]])
        v = np.concatenate([rng.integers(0, n, k).astype(np.uint32), d[e]])
        x = np.concatenate([rng.uniform(0.5, 2.0, k), -w[e]])
        ref = g.apply_delta(u, v, x, keep_self_loops=True)
        got = gh.apply_delta(g, u, v, x, keep_loops=True)
        for a, b in zip(got, ref.csr()):
            assert gh.same_bits(a, b)
    # and weight changes alone, which need no second buffer
    ref = g.apply_delta(s[:500], d[:500], np.ones(500), keep_self_loops=True)
    got = gh.apply_delta(g, s[:500], d[:500], np.ones(500), keep_loops=True)
    for a, b in zip(got, ref.csr()):
        assert gh.same_bits(a, b)


# A few seeds wake the whole level: a launch whose blocks were chosen for the
# seeds hands over to one with more of them, from one block and from a cluster.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("n,m", [(900, 3000), (1500, 60000), (20000, 160000)])
def test_frontier_outgrows_its_launch(n, m, integral):
    rng = np.random.default_rng(n)
    s, d, w = gh.random_graph(rng, n, m, integral)
    g = O.Graph.from_edges(n, s, d, w).apply_delta([], [], [], keep_self_loops=True)
    f = np.arange(n, dtype=np.uint32)
    sub = gh.random_partition(rng, n, n // 3)
    delta = s[:2], d[:2], np.ones(2)
    for rounds in (1, 4, 20):
        ref = O.inc_movement(g, *delta, f.copy(), sub, 1.0, O.MODE_THROUGHPUT, max_rounds=rounds)
        got = gh.inc_movement(g, *delta, f, sub, 1.0, max_rounds=rounds)
        assert ref[3] == got[3] and all(np.array_equal(ref[i], got[i]) for i in range(3))
    assert ref[1].sum() > n // 2  # most vertices have moved


# Hub rows side by side, in a batch above the one-launch limit: their sums run
# beside each other (one warp took 32 rows in turn: 4.5 ms here with f64
# weights).  Same bits as the oracle's CSR and degrees.
@pytest.mark.parametrize("integral", [True, False])
def test_adjacent_hub_rows(integral):
    rng = np.random.default_rng(5)
    n, hubs, deg = 30000, 64, 20000
    s = np.repeat(np.arange(hubs, dtype=np.uint32), deg)
    d = np.concatenate([rng.choice(np.arange(hubs, n), deg, replace=False)
                        for _ in range(hubs)]).astype(np.uint32)
    w = np.ones(len(s)) if integral else rng.uniform(0.5, 2.0, len(s))
    gs = _load(n, (s, d, w), max_iterations=1, kernel_timing=True)
    ref = O.State(n, levels=1, mode=O.MODE_THROUGHPUT)
    ref.push_empty_graph()
    ref.hit_leiden(s, d, w)
    e = rng.choice(len(s), 40000, replace=False)
    b = s[e], d[e], np.ones(len(e)) if integral else rng.uniform(0.5, 2.0, len(e))
    gs.apply_batch(*b)
    before = gs.kernel_stats()["row_sums"]
    gs.apply_batch(*b)
    after = gs.kernel_stats()["row_sums"]
    ref.hit_leiden(*b)
    ref.hit_leiden(*b)
    _same(gs, ref)
    off, col, wt = gs.supergraph(0)
    ro, rc, rw = ref.graph(0).csr()
    assert np.array_equal(off, ro) and np.array_equal(col, rc) and gh.same_bits(wt, rw)
    assert gs.modularity() == pytest.approx(ref.modularity(0), abs=1e-12)
    assert after["launches"] - before["launches"] == 1
    assert after["ms"] - before["ms"] < 1.0, after["ms"] - before["ms"]
    gs.close()


# Two hubs whose half a million leaves each are split and merged again: the
# upper level's edges are sums of half a million records each, which must not
# wait for one another.
@pytest.mark.parametrize("integral", [True, False])
def test_long_segments_of_the_aggregation(integral):
    n, edges = _double_star(500000, integral)
    gs, ref = _load(n, edges), _oracle(n, edges)
    b = np.array([2], np.uint32), np.array([3], np.uint32), np.ones(1)
    gs.apply_batch(*b)
    ref.hit_leiden(*b)
    _same(gs, ref)
    for p in range(ref.levels):
        off, col, wt = gs.supergraph(p)
        ro, rc, rw = ref.graph(p).csr()
        assert np.array_equal(off, ro) and np.array_equal(col, rc) and gh.same_bits(wt, rw)
    gs.close()


# Long ordered sums choose a fold every 65,536 terms by the signs they meet, and
# one addition after another below 16,384: at and around both lengths, sums that
# change sign inside a piece and at its edge, zeros and values that are not
# finite.  All three paths, bit for bit.
@pytest.mark.parametrize("kind", ["positive", "negative", "late", "edge", "mixed", "zeros", "inf"])
def test_long_sums_choose_their_fold(kind):
    rng = np.random.default_rng(len(kind))
    segs = []
    for n in (16383, 16384, 16385, 65536, 65537, 81919, 81920, 150001):
        x = rng.uniform(0.5, 60.0, n)
        if kind == "negative":
            x = -x
        elif kind == "late":  # after the first terms that are looked at
            x[100::7] *= -3.0
        elif kind == "edge":
            x[65536:] *= -1.0
        elif kind == "mixed":
            x[::2] *= -1.0
        elif kind == "zeros":
            x[rng.random(n) < 0.9] = 0.0
        elif kind == "inf":
            x[n // 2] = np.inf
        segs.append(x)
    L = gh.L
    off = np.concatenate([[0], np.cumsum([len(s) for s in segs])]).astype(np.uint64)
    x = np.concatenate(segs)
    want = np.array([np.cumsum(np.concatenate([[0.0], s]))[-1] for s in segs])
    for path in (0, 1, 2):
        got = np.zeros(len(segs))
        L.check(L.lib.hl_dbg_seq_sums(0, len(segs), L.ptr(off), L.ptr(x), 0.0, path, L.ptr(got)))
        assert gh.same_bits(got, want), (kind, path)


# Tags and reservation keys of earlier selections stay in memory.  When their
# counters start again, a batch must not read them as its own: round numbers
# repeat those of the batches before.  One-launch rounds and multi-kernel ones.
@pytest.mark.parametrize("integral", [True, False])
@pytest.mark.parametrize("multi", [False, True])
def test_selection_counters_start_again(integral, multi):
    rng = np.random.default_rng(11 + integral)
    n = 3000
    edges = gh.random_graph(rng, n, 9000, integral)
    gs = _load(n, edges, small_rounds=not multi)
    ref = _oracle(n, edges)
    L = gh.L
    for i in range(6):
        b = _updates(rng, n, edges, 300, integral)
        if i >= 2:  # near the end of the tags, near the end of the epochs
            at = ((1 << 29) - 3, 1 << 20) if i % 2 else (7, (1 << 31) + 5)
            L.check(L.lib.hl_dbg_set_selection(gs._h, *at))
        gs.apply_batch(*b)
        ref.hit_leiden(*b)
        _same(gs, ref)
    gs.close()


# A movement that never settles: several launches of the one-launch rounds, with
# a multi-kernel round between them, up to the cap.
@pytest.mark.parametrize("cap", [1023, 1024, 1025, 1026, 3000])
def test_rounds_past_one_launch(cap):
    rng = np.random.default_rng(69)
    n = int(rng.integers(6, 120))
    m = int(n * rng.uniform(1, 8))
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    s, d = s[s != d], d[s != d]
    g = O.Graph.from_edges(n, s, d, np.ones(len(s)))
    ident = np.arange(n, dtype=np.uint32)
    ref = O.inc_movement(g, [], [], [], ident.copy(), ident, 2.0, O.MODE_THROUGHPUT, max_rounds=cap)
    got = gh.inc_movement(g, [], [], [], ident, ident, 2.0, max_rounds=cap)
    assert ref[3] == cap and got[3] == cap
    assert all(np.array_equal(ref[i], got[i]) for i in range(3))


# "No cap" on the movement rounds: every u32 is a valid max_rounds.  These
# movements end by themselves after a few dozen rounds.
@pytest.mark.parametrize("max_rounds", [1 << 20, 10 ** 9, (1 << 32) - 1])
def test_uncapped_rounds(max_rounds):
    n, s, d, w, _ = W.planted(3000, 8.0, 0.1, 5, comm_min=8, comm_max=60, triangle_frac=0.3)
    rng = np.random.default_rng(3)
    w = rng.uniform(0.5, 2.0, len(s))
    ref = _oracle(n, (s, d, w), max_rounds=max_rounds)
    gs = _load(n, (s, d, w), max_rounds=max_rounds)
    _same(gs, ref)
    for _ in range(4):
        b = _updates(rng, n, (s, d, w), 100, False)
        gs.apply_batch(*b)
        ref.hit_leiden(*b)
        _same(gs, ref)
    gs.close()


# A program's exit handler destroys handles after the library's own statics are
# gone: the pool their staging blocks go back to must still be there (an abort
# of the program on a second free otherwise).
def test_handles_outlive_static_destruction(tmp_path):
    import shutil
    import subprocess
    from pathlib import Path
    root = Path(hl.__file__).resolve().parents[1]
    gcc = shutil.which("gcc")
    if gcc is None:
        pytest.skip("no C compiler")
    src = tmp_path / "late.c"
    src.write_text("""
#include <stdlib.h>
#include "hl.h"
static hl_graph* g[3];
static void bye(void) { hl_destroy(g[1]); hl_destroy(g[2]); }
int main(void) {
  uint32_t u[3] = {0, 1, 2}, v[3] = {1, 2, 3};
  hl_config c;
  hl_config_default(&c);
  if (atexit(bye)) return 3;
  for (int i = 0; i < 3; ++i)
    if (hl_create(&c, 4, u, v, 0, 3, &g[i]) != HL_OK) return 2;
  hl_destroy(g[0]);
  return 0;
}
""")
    exe = tmp_path / "late"
    lib = Path(hl.__file__).resolve().parent / "libhl.so"
    subprocess.run([gcc, "-I", str(root / "include"), str(src), str(lib), "-o", str(exe),
                    f"-Wl,-rpath,{lib.parent}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)
