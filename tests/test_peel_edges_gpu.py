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
