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


# "No cap" on the movement rounds: every u32 is a valid max_rounds.  These
# movements end by themselves after a few dozen rounds.
@pytest.mark.parametrize("max_rounds", [(1 << 24) + 1, 10 ** 9, (1 << 32) - 1])
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
