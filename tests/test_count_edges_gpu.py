"""The warp, mid and block aggregators at the edges of their tables: wedge counts around the limits
of each class, counts that fill a one-word entry's or a 16-bit counter's neighbourhood, rows longer
than a warp or a mid CTA takes, and the lowest ranks gathered per CTA."""
import numpy as np
import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200.graph import BipartiteGraph

pytestmark = pytest.mark.gpu


def _biclique(a, b, extra=0, seed=1, isolated=0):
    """K_{a,b} and `extra` random edges on an (a + isolated) x (b + isolated) grid."""
    rng = np.random.default_rng(seed)
    v = np.r_[np.repeat(np.arange(a), b), rng.integers(0, a + isolated, extra)]
    u = np.r_[np.tile(np.arange(b), a), rng.integers(0, b + isolated, extra)]
    return BipartiteGraph.from_edges(a + isolated, b + isolated, v, u)


GRAPHS = {
    # Endpoint wedge counts of 1 .. a * b around 512 (warp / mid) and 2047 (mid / block).
    "k23_23": lambda: _biclique(23, 23),
    "k46_46": lambda: _biclique(46, 46),
    "k17_700": lambda: _biclique(17, 700, 3000, 2, 500),
    # Rows of 1023 .. 1025 and 16385 slots with few wedges each.
    "rows": lambda: BipartiteGraph.from_edges(
        40_000, 6, np.r_[np.arange(1023), np.arange(1024), np.arange(1025), np.arange(16_385), 39_998, 39_999],
        np.r_[np.zeros(1023, int), np.ones(1024, int), np.full(1025, 2), np.full(16_385, 3), 4, 5]),
    # Rows of 255 .. 257 slots, the first length of the small CTAs.
    "rows_256": lambda: BipartiteGraph.from_edges(
        3_000, 5, np.r_[np.arange(255), np.arange(256), np.arange(257), 2_998, 2_999],
        np.r_[np.zeros(255, int), np.ones(256, int), np.full(257, 2), 3, 4]),
    # More vertices than leave ten count bits beside a key: two-array tables.
    "many_vertices": lambda: _biclique(30, 600, 60_000, 3, 2_200_000),
    # Prefixes on both sides of the length that all warps of a CTA walk together.
    "long_prefix": lambda: _biclique(5, 1500, 20_000, 4, 3000),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_aggregator_limits(ctx, name):
    g = GRAPHS[name]()
    dg = ctx.upload(g)
    for rank in ["ADEG", "SIDE"]:
        want_v, want_e = oracle.count(g, "VERT", rank)[0], oracle.count(g, "EDGE", rank)[0]
        assert np.array_equal(pb.count(dg, "BATCHS", rank), want_v)
        assert np.array_equal(pb.count_e(dg, "HASH", rank), want_e)
        assert pb.count_total(dg, "SERIAL", rank) == int(want_v.sum()) // 2
        other = not pb.cmp_wedge_counts(dg)[0]
        assert np.array_equal(pb.count(dg, "BATCHS", rank, use_v=other), oracle.count(g, "VERT", rank, use_v=other)[0])
    dg.close()


def test_degrees_beyond_16_bits(ctx):
    """An endpoint of more than 65535 neighbours shares more than 65535 of them with another: dense
    counters and hash entries fall back to 32 bits."""
    n = 66_000
    g = BipartiteGraph.from_edges(n, 300, np.r_[np.arange(n), np.arange(n), np.arange(3, 900) % 50],
                                  np.r_[np.zeros(n, int), np.ones(n, int), np.arange(3, 900) % 297 + 3])
    dg = ctx.upload(g)
    for use_v in (False, True):
        assert np.array_equal(pb.count(dg, "BATCHS", "SIDE", use_v=use_v), oracle.count(g, "VERT", "SIDE", use_v=use_v)[0])
        assert np.array_equal(pb.count_e(dg, "HASH", "SIDE", use_v=use_v), oracle.count(g, "EDGE", "SIDE", use_v=use_v)[0])
    dg.close()


@pytest.mark.parametrize("rows", [300, 512, 513, 1100])
def test_lists_beside_a_warps_share(ctx, rows):
    """Dense rows of lists that a warp each walks, lists of all warps among them: the limit between the
    two lies at a quarter of a warp's share of the row's chunk."""
    hub = 20_000
    g = BipartiteGraph.from_edges(rows + 2, hub, np.r_[np.repeat(np.arange(rows), 700), np.full(hub, rows),
                                                       np.full(hub // 2, rows + 1)],
                                  np.r_[np.tile(np.arange(700), rows), np.arange(hub), np.arange(0, hub, 2)])
    dg = ctx.upload(g)
    for rank in ["SIDE", "DEG"]:
        for use_v in (False, True):
            assert np.array_equal(pb.count(dg, "BATCHS", rank, use_v=use_v), oracle.count(g, "VERT", rank, use_v=use_v)[0])
        assert np.array_equal(pb.count_e(dg, "HASH", rank), oracle.count(g, "EDGE", rank)[0])
    dg.close()
