"""Peel rounds at the edges of the schedules a round can take: frontiers whose two-hop lists add up to
the limit of the list-per-warp pass and beyond it, more heavy items than one or two waves hold, and
wing frontiers around the largest one-slice-per-CTA round.  Every vertex (edge) of a complete
bipartite graph has the same count, so its whole side (all its edges) is one round."""
import numpy as np
import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200.graph import BipartiteGraph

pytestmark = pytest.mark.gpu


def _bicliques(*sizes, extra=0, seed=1):
    """Disjoint K_{a,b} for every (a, b), and `extra` random edges over all of it."""
    v, u, v0, u0 = [], [], 0, 0
    for a, b in sizes:
        v.append(np.repeat(np.arange(a), b) + v0)
        u.append(np.tile(np.arange(b), a) + u0)
        v0, u0 = v0 + a, u0 + b
    rng = np.random.default_rng(seed)
    v.append(rng.integers(0, v0, extra))
    u.append(rng.integers(0, u0, extra))
    return BipartiteGraph.from_edges(v0, u0, np.concatenate(v), np.concatenate(u))


@pytest.mark.parametrize("sizes,extra", [
    ([(128, 16)], 0),                 # 16 items, 2^15 pairs: list per warp
    ([(129, 16)], 0),                 # 2^15 + 256 pairs: equal slices
    ([(300, 32), (300, 33)], 0),      # 32 and 33 heavy items
    ([(100, 100), (100, 100)], 0),    # 200 heavy items in one round: two waves
    ([(90, 96)] * 3, 40),             # three waves, then ragged rounds
    ([(16, 128), (40, 7), (7, 40)], 300),
])
def test_tip_rounds(ctx, sizes, extra):
    g = _bicliques(*sizes, extra=extra)
    dg = ctx.upload(g)
    for use_v in (False, True):
        c = pb.count(dg, "BATCHS", "ADEG", use_v=use_v)
        want = oracle.peel_vert(g, c, use_v=use_v)[0]
        for parts in (0, 3):
            assert np.array_equal(pb.peel(dg, c, use_v=use_v, peel_parts=parts), want)
    dg.close()


@pytest.mark.parametrize("small_work", ["0", "512"])
@pytest.mark.parametrize("sizes,extra", [
    ([(2, 37)], 0), ([(5, 15)], 0),              # 74 and 75 edges in one round (148 CTAs)
    ([(8, 16)], 0), ([(3, 43)], 0),              # 128 and 129
    ([(32, 40), (33, 41)], 0),                   # first levels of 32 and 33 entries
    ([(3, 270), (270, 3), (20, 20)], 500),       # probe sets around a warp table's 256 entries
])
def test_wing_rounds(ctx, monkeypatch, sizes, extra, small_work):
    monkeypatch.setenv("PB_PEEL_SMALL_WORK", small_work)
    g = _bicliques(*sizes, extra=extra)
    dg = ctx.upload(g)
    for use_v in (False, True):
        c = pb.count_e(dg, "HASH", "ADEG", use_v=use_v)
        assert np.array_equal(pb.peel_e(dg, c, use_v=use_v), oracle.peel_edge(g, c, use_v=use_v)[0])
    dg.close()


def _hubs(n, h, m, seed):
    rng = np.random.default_rng(seed)
    return BipartiteGraph.from_edges(n, n, np.r_[np.repeat(np.arange(h), n), rng.integers(0, n, m)],
                                     np.r_[np.tile(np.arange(n), h), rng.integers(0, n, m)])


@pytest.mark.parametrize("graph", [
    lambda: _hubs(6000, 4, 40_000, 3),                      # most work with probe sets above 4,096 entries
    lambda: _hubs(4096, 5, 30_000, 4),                      # probe sets of 4,096
    lambda: BipartiteGraph.uniform(700, 500, 32_768, 5),    # even work, at and above the size from which it is looked at
    lambda: BipartiteGraph.uniform(700, 500, 32_769, 5),
])
def test_wing_kernels_of_one_and_two_ctas(ctx, graph):
    g = graph()
    dg = ctx.upload(g)
    c = pb.count_e(dg, "HASH", "ADEG")
    assert np.array_equal(pb.peel_e(dg, c), oracle.peel_edge(g, c)[0])
    dg.close()


def test_wing_hubs_run_two_ctas_per_sm(ctx, monkeypatch):
    """Hubs whose lists exceed shared memory: probes wait for device memory, so a CTA per SM (forced below) is
    too few (39.7 ms against 26.4)."""
    import torch
    dg = ctx.upload(_hubs(20_000, 4, 100_000, 5))
    c = pb.count_e(dg, "HASH", "ADEG")

    def best():
        runs = [(pb.peel_e(dg, c), ctx.stats()["ms_peel"]) for _ in range(4)]
        return runs[0][0], min(t for _, t in runs)

    out, ms = best()
    monkeypatch.setenv("PB_PEEL_CTAS", str(torch.cuda.get_device_properties(0).multi_processor_count))
    out_one, ms_one = best()
    assert np.array_equal(out, out_one)
    assert ms < 0.85 * ms_one
    dg.close()


@pytest.mark.parametrize("few", [1, 8, 31, 32, 33, 63, 64])
def test_tip_of_few_vertices(ctx, few):
    """A handful of heavy vertices against many: slices of counters around multiples of a memory line, and
    waves of all vertices."""
    g = BipartiteGraph.uniform(few, 3000, 1500 * few, 12)
    dg = ctx.upload(g)
    for use_v in (False, True):
        c = pb.count(dg, "BATCHS", "ADEG", use_v=use_v)
        want = oracle.peel_vert(g, c, use_v=use_v)[0]
        for parts in (0, 3):
            assert np.array_equal(pb.peel(dg, c, use_v=use_v, peel_parts=parts), want)
    dg.close()
