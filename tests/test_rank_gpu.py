"""The ranked CSR at the edges of its builders: slots around the line between the row sort and the
radix sort, rows that begin and end inside a 256-slot chunk, long runs of empty rows, and co-core
ranking with lists around multiples of its 256-entry units.  The order is checked through the ranked
wedge count (equal to the oracle's only for the same order), the rows through the counts."""
import numpy as np
import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200.graph import BipartiteGraph

pytestmark = pytest.mark.gpu


def _hubs():
    """Stars of 255, 256, 257, 512 and 513 leaves that share leaves, and isolated vertices between."""
    v, u = [], []
    for k, d in enumerate((255, 256, 257, 512, 513)):
        v.append(np.full(d, 40 * k))
        u.append(np.arange(d) * 3)
    return BipartiteGraph.from_edges(400, 2000, np.concatenate(v), np.concatenate(u))


GRAPHS = {
    "slots_below": lambda: BipartiteGraph.uniform(9_000, 7_000, (1 << 18) - 1, 31),
    "slots_at": lambda: BipartiteGraph.rmat(14, 12, 1 << 18, 0.55, 0.15, 0.15, 0.15, 32),
    "slots_above": lambda: BipartiteGraph.powerlaw_u(5_000, 30_000, (1 << 18) + 1, 2.0, 5_000, 33),
    "one_tile": lambda: BipartiteGraph.uniform(2_000, 2_096, 9_000, 35),    # 4096 vertices: one radix tile
    "two_tiles": lambda: BipartiteGraph.uniform(2_000, 2_097, 9_000, 36),
    "search_below": lambda: BipartiteGraph.uniform(3_000, 2_000, (1 << 17) + 1, 37),  # 2^18 + 2 slots
    "hubs": _hubs,
    "sparse": lambda: BipartiteGraph.uniform(200_000, 150_000, 3_000, 34),
    "one_row": lambda: BipartiteGraph.from_edges(3, 700, np.r_[np.zeros(700, int), 1, 1], np.r_[np.arange(700), 0, 699]),
}


@pytest.mark.parametrize("rank", ["SIDE", "COCORE", "ACOCORE", "DEG", "ADEG"])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_ranked_csr(ctx, name, rank):
    g = GRAPHS[name]()
    dg = ctx.upload(g)
    want, w_rank = oracle.count(g, "VERT", rank)
    assert np.array_equal(pb.count(dg, "HASH", rank), want)
    assert ctx.stats()["w_rank"] == w_rank
    assert np.array_equal(pb.count_e(dg, "BATCHS", rank), oracle.count(g, "EDGE", rank)[0])
    dg.close()


@pytest.mark.parametrize("rank", ["SIDE", "COCORE", "ACOCORE"])
def test_long_runs_of_empty_rows(ctx, rank):
    """Millions of vertices without edges between two slots: the rows are found by a search, not by
    walking through the run (which took the two stages 70 ms each on this graph)."""
    n, rng = 1 << 22, np.random.default_rng(39)

    def ids():
        x = rng.integers(0, 3_000, 20_000)
        return np.where(x < 1_500, x, np.where(x < 1_700, 100_000 + 37 * x, n - 1 - x))

    g = BipartiteGraph.from_edges(n, n, ids(), ids())
    dg = ctx.upload(g)
    want = oracle.count(g, "VERT", rank)[0]
    for _ in range(2):
        assert np.array_equal(pb.count(dg, "HASH", rank), want)
    st = ctx.stats()
    assert st["ms_relabel"] + st["ms_scan"] < 14.0
    assert np.array_equal(pb.count_e(dg, "SORT", rank), oracle.count(g, "EDGE", rank)[0])
    dg.close()


@pytest.mark.parametrize("a,b", [(1000, 1000), (257, 8000)])
def test_few_vertices_with_long_lists(ctx, a, b):
    """The lists of a few vertices are spread over the device, not over the CTAs that hold a thread per
    vertex (the 8,000 units of K_{1000,1000} took two CTAs 0.48 ms; spread, 0.08)."""
    g = BipartiteGraph.from_edges(a, b, np.repeat(np.arange(a), b), np.tile(np.arange(b), a))
    dg = ctx.upload(g)
    ms = []
    for rank in ["ACOCORE", "COCORE"] * 4:
        assert pb.count_total(dg, "HASH", rank) == (a * (a - 1) // 2) * (b * (b - 1) // 2)
        ms.append(ctx.stats()["ms_rank"])
    assert min(ms) < 0.25
    dg.close()


def test_barrier_timeout_reports_status_and_context_survives(ctx, monkeypatch):
    """A barrier wait of the co-core ranking that cannot complete (test hook) runs out after the
    configured bound: single calls and replays of a captured batch return PB_ETIMEOUT."""
    from parbutterfly_b200._ffi import PB_ETIMEOUT, PBError
    g = BipartiteGraph.zipf(3_000, 4_000, 30_000, 1.3, 38)
    dg = ctx.upload(g)
    want = oracle.count(g, "VERT", "ACOCORE")[0]
    tips = oracle.peel_vert(g, want)[0]
    monkeypatch.setenv("PB_RANK_BARRIER_TIMEOUT_MS", "300")
    monkeypatch.setenv("PB_RANK_TEST_STUCK_BARRIER", "1")
    with pytest.raises(PBError) as ex:
        pb.count(dg, "HASH", "ACOCORE")
    assert ex.value.status == PB_ETIMEOUT
    monkeypatch.setenv("PB_RANK_TEST_STUCK_BARRIER", "2")
    batch = pb.BatchGraph([dg, dg], rank_type="ACOCORE")
    for _ in range(2):
        with pytest.raises(PBError) as ex:
            batch.run()
        assert ex.value.status == PB_ETIMEOUT
    batch.close()
    monkeypatch.delenv("PB_RANK_TEST_STUCK_BARRIER")
    assert np.array_equal(pb.count(dg, "HASH", "ACOCORE"), want)
    batch = pb.BatchGraph([dg, dg], rank_type="ACOCORE")
    for _ in range(2):
        c, t = batch.run()
        assert all(np.array_equal(x, want) for x in c) and all(np.array_equal(x, tips) for x in t)
    batch.close()
    dg.close()
