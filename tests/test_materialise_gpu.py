"""SORT / HIST at the edges of the materialised path: 32-bit against 64-bit wedge keys (the key
holds the batch's endpoints and the vertex ids), one batch against several, long runs of slots
without wedges, chunks that end inside a slot."""
import numpy as np
import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200.graph import BipartiteGraph

pytestmark = pytest.mark.gpu

GRAPHS = {
    "keys32": lambda: BipartiteGraph.uniform(30_000, 35_000, 200_000, 11),        # 16 + 16 bits
    "keys33": lambda: BipartiteGraph.uniform(30_000, 36_000, 200_000, 12),        # 17 + 17 bits
    "hub": lambda: BipartiteGraph.from_edges(                                      # one slot of 3000 wedges
        40, 3000, np.r_[np.zeros(3000, int), np.ones(2999, int), np.arange(2, 40)],
        np.r_[np.arange(3000), np.arange(1, 3000), np.arange(2, 40)]),
    "few": lambda: BipartiteGraph.from_edges(50_000, 50_000, np.r_[np.arange(49_998), 49_998, 49_998, 49_999, 49_999],
                                             np.r_[np.arange(49_998), 49_998, 49_999, 49_998, 49_999]),  # 1 butterfly
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("count_type", ["SORT", "HIST"])
@pytest.mark.parametrize("max_wedges", [2577500000, 1000])
def test_materialised_counts(ctx, name, count_type, max_wedges):
    g = GRAPHS[name]()
    dg = ctx.upload(g)
    for per, fn in [("VERT", pb.count), ("EDGE", pb.count_e)]:
        want, _ = oracle.count(g, per, "ADEG")
        if max_wedges == 1000 and len(want) > 10_000 and name.startswith("keys"):
            continue  # thousands of batches
        assert np.array_equal(fn(dg, count_type, "ADEG", max_wedges=max_wedges), want)
    total = int(oracle.count(g, "VERT", "ADEG")[0].sum()) // 2
    assert pb.count_total(dg, count_type, "SIDE") == total
    dg.close()
