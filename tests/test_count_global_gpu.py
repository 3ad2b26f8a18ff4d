"""The global-scratch mode of the CTA aggregator over many endpoints in a row: the counters that an
endpoint leaves behind must be zero when its CTA takes the next one.  Rows span several chunks of
512 slots, so the walks that count, credit and clear follow each other with short and long chunks."""
import numpy as np
import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200.graph import BipartiteGraph

pytestmark = pytest.mark.gpu

GLOBAL = 12 + 2  # a trace row's features are followed by the one-hot mode: dense, hash, global, hybrid


def _heavy_tail():
    """600 count-side vertices of about 1100 neighbours behind 4500 of one: beyond every table of 16 KiB."""
    rng = np.random.default_rng(6)
    heavy = np.repeat(np.arange(4500, 5100), 1400)
    return BipartiteGraph.from_edges(3000, 5100, np.r_[rng.integers(0, 3000, 4500), rng.integers(0, 3000, heavy.size)],
                                     np.r_[np.arange(4500), heavy])


@pytest.mark.parametrize("make,rank,use_v", [
    (_heavy_tail, "SIDE", True),                                             # endpoint and edge credits
    (lambda: BipartiteGraph.uniform(3000, 3000, 1_900_000, 7), "DEG", True),  # centre credits as well
])
def test_many_global_endpoints_per_cta(ctx, monkeypatch, make, rank, use_v):
    monkeypatch.setenv("PB_COUNT_SMEM", "16384")
    monkeypatch.setenv("PB_COUNT_BPS", "1")
    g = make()
    dg = ctx.upload(g)
    want_v = oracle.count(g, "VERT", rank, use_v=use_v)[0]
    want_e = oracle.count(g, "EDGE", rank, use_v=use_v)[0]
    for _ in range(5):
        assert np.array_equal(pb.count(dg, "BATCHS", rank, use_v=use_v), want_v)
        assert np.array_equal(pb.count_e(dg, "HASH", rank, use_v=use_v), want_e)
    pb.trace_set(ctx, "plain")
    try:
        pb.trace_clear(ctx)
        pb.count_e(dg, "HASH", rank, use_v=use_v)
        rows, _ = pb.trace_rows(ctx, pb.SchedModel.COUNT)
    finally:
        pb.trace_set(ctx, "off")
        pb.trace_clear(ctx)
    assert rows[:, GLOBAL].sum() > 3 * 148  # several per CTA
    dg.close()
