"""Device memory that calls take beside their inputs and outputs: graphs of many vertices and few
edges, where arrays per vertex decide, and calls that must get by with what is left of a device."""
import ctypes as C

import numpy as np
import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200.graph import BipartiteGraph

pytestmark = pytest.mark.gpu

USED_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


class _Pool:
    """The device's default memory pool, from which the library allocates."""

    def __init__(self):
        import torch
        torch.cuda.init()
        self.cu = C.CDLL("libcuda.so.1")
        self.pool = C.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), 0) == 0

    def reset(self):
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(C.c_uint64(0))) == 0
        return self.high()

    def high(self):
        x = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, USED_HIGH, C.byref(x)) == 0
        return x.value

    def trim(self):
        assert self.cu.cuMemPoolTrimTo(self.pool, C.c_size_t(0)) == 0


@pytest.fixture(scope="module")
def pool():
    return _Pool()


def _spread(nu, k, nv, deg, seed):
    """k U-vertices spread over [0, nu), each with `deg` draws of nv V-vertices: the graph on the GPU, the
    same graph without the isolated U-vertices, and the U-vertices' ids."""
    import torch
    rng = np.random.default_rng(seed)
    ids = np.unique(np.r_[0, nu - 1, rng.integers(0, nu, k)])
    small = BipartiteGraph.from_edges(nv, ids.size, rng.integers(0, nv, ids.size * deg), np.repeat(np.arange(ids.size), deg))
    at = torch.from_numpy(ids).cuda()
    deg_u = torch.zeros(nu + 1, dtype=torch.int64, device="cuda")
    deg_u[at + 1] = torch.from_numpy(np.diff(small.offsetsU.astype(np.int64))).cuda()
    off_u = torch.cumsum(deg_u, 0).to(torch.int32)
    del deg_u
    off_v, edg_u = (torch.from_numpy(a.astype(np.int32)).cuda() for a in (small.offsetsV, small.edgesU))
    edg_v = at[torch.from_numpy(small.edgesV.astype(np.int64)).cuda()].to(torch.int32)
    torch.cuda.synchronize()
    return (nv, nu, off_v, edg_v, off_u, edg_u), small, at


def test_count_lists_of_many_vertices(ctx, pool):
    """Endpoints in three stretches of the ranks; item lists for all vertices at once would take 48 bytes
    each."""
    import torch
    nu = (1 << 27) + 12_345
    arrays, small, at = _spread(nu, 40_000, 1000, 5, 1)
    dg = pb.DeviceGraph(ctx, device_arrays=arrays)
    del arrays
    base = pool.reset()
    out = torch.zeros(nu, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    pb.count(dg, "BATCHS", "SIDE", use_v=True, out=out)
    assert pool.high() - base < 56 * nu  # 28 for the ranking and the sums, 24 for lists of 2^26 endpoints
    assert np.array_equal(out[at].cpu().numpy(), oracle.count(small, "VERT", "SIDE", use_v=True)[0])
    assert int(torch.count_nonzero(out)) == int(torch.count_nonzero(out[at]))
    assert np.array_equal(pb.count_e(dg, "HASH", "SIDE", use_v=True), oracle.count(small, "EDGE", "SIDE", use_v=True)[0])
    assert pb.count_total(dg, "SERIAL", "SIDE", use_v=True) == oracle.count(small, "TOTAL", "SIDE", use_v=True)[0]
    dg.close()


@pytest.mark.parametrize("parts", [0, 4])
def test_tip_lists_of_many_vertices(ctx, pool, parts):
    """Descriptors of heavy items are kept for the vertices that can be heavy, not for all."""
    import torch
    nu = (1 << 27) + 12_345
    arrays, small, at = _spread(nu, 4_000, 300, 5, 2)
    dg = pb.DeviceGraph(ctx, device_arrays=arrays)
    del arrays
    out = torch.zeros(nu, dtype=torch.int64, device="cuda")
    counts = torch.zeros_like(out)
    torch.cuda.synchronize()
    pb.count(dg, "BATCHS", "ADEG", use_v=True, out=counts)
    base = pool.reset()
    pb.peel(dg, counts, use_v=True, out=out, peel_parts=parts)
    # Lists, frontiers, counts, work and states: 61 bytes; batched rounds 16 (opening counts,
    # partitions, weights) and 16 (sorted items) more; grid-shared counters 2 GiB.
    assert pool.high() - base < (64 if parts == 0 else 96) * nu + (2 << 30) + (64 << 20)
    want = oracle.peel_vert(small, oracle.count(small, "VERT", "ADEG", use_v=True)[0], use_v=True)[0]
    assert np.array_equal(out[at].cpu().numpy(), want)
    assert int(torch.count_nonzero(out)) == int(np.count_nonzero(want))
    dg.close()


@pytest.fixture
def short_of_memory(pool):
    """leave(n): takes the device's memory until n bytes are left."""
    import torch
    held = []

    def leave(n):
        torch.cuda.synchronize()
        pool.trim()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        if free < n:
            pytest.skip("less memory free than the call needs")
        held.append(torch.empty(free - n, dtype=torch.uint8, device="cuda"))

    yield leave
    held.clear()
    torch.cuda.empty_cache()


def test_batched_tip_rounds_short_of_memory(ctx, pool, short_of_memory):
    """Dense counters of one CTA per SM fit what is left (9.9 GB), those of two do not."""
    import torch
    arrays, small, _ = _spread(1 << 24, 40_000, 30, 3, 3)
    dg = pb.DeviceGraph(ctx, device_arrays=arrays)
    del arrays
    out = torch.zeros(1 << 24, dtype=torch.int64, device="cuda")
    counts = torch.zeros_like(out)
    torch.cuda.synchronize()
    pb.count(dg, "BATCHS", "ADEG", use_v=True, out=counts)
    short_of_memory(17 << 30)
    pb.peel(dg, counts, use_v=True, out=out, peel_parts=4)
    want = oracle.peel_vert(small, oracle.count(small, "VERT", "ADEG", use_v=True)[0], use_v=True)[0]
    got = out.cpu().numpy()
    assert np.array_equal(got[got > 0], want[want > 0])
    dg.close()


def test_relabel_short_of_memory(ctx, pool, short_of_memory):
    """A per-edge count of 2^26 edges needs 3.0 GB beside the graph when rows are sorted in place, 3.9 GB
    when the slots are sorted as a whole; with 3.45 GB left it takes the first way."""
    _check_shifts(ctx, short_of_memory, 3450 << 20)


@pytest.mark.parametrize("acc64", [False, True])
def test_edge_credits_short_of_memory(ctx, pool, short_of_memory, monkeypatch, acc64):
    """The same count with 2.7 GB left: 2.4 GB are needed without counts per slot, 3.0 or 3.5 with them."""
    if acc64:
        monkeypatch.setenv("PB_EDGE_ACC64", "1")
    _check_shifts(ctx, short_of_memory, 2600 << 20)


def _check_shifts(ctx, short_of_memory, left):
    import torch
    n, d = 1 << 21, 32  # v's neighbours are v + 127 j, so u's are u - 127 j
    v = torch.arange(n, device="cuda").unsqueeze(1)
    j = 127 * torch.arange(d, device="cuda").unsqueeze(0)
    edg_v = torch.sort((v + j) % n, 1)[0].to(torch.int32).reshape(-1)
    edg_u = torch.sort((v - j) % n, 1)[0].to(torch.int32).reshape(-1)
    off = (d * torch.arange(n + 1, device="cuda")).to(torch.int32)
    torch.cuda.synchronize()
    dg = pb.DeviceGraph(ctx, device_arrays=(n, n, off, edg_v, off, edg_u))
    del edg_v, edg_u, off, v, j
    short_of_memory(left)
    got = pb.count_e(dg, "HASH", "SIDE").reshape(n, d)
    # v and v + 127 t share d - |t| neighbours.
    want = np.array([sum(d - 1 - abs(j - k) for k in range(d) if k != j) for j in range(d)])
    assert (got[:n - 127 * d] == want).all() and int(got.sum()) == n * int(want.sum())
    dg.close()


def test_tip_counters_follow_the_peeled_side(ctx, pool):
    """Few vertices peeled against many: the heavy items' counters are slices of the peeled side (slices of
    the longer one took 512 bytes a centre)."""
    nv, nu = 400_000, 40
    rng = np.random.default_rng(8)
    g = BipartiteGraph.from_edges(nv, nu, rng.integers(0, nv, 1_000_000), rng.integers(0, nu, 1_000_000))
    dg = ctx.upload(g)
    counts = pb.count(dg, "BATCHS", "ADEG", use_v=True)
    want = oracle.peel_vert(g, counts)[0]
    for parts in (0, 8):
        base = pool.reset()
        assert np.array_equal(pb.peel(dg, counts, peel_parts=parts), want)
        assert pool.high() - base < 128 * nv
    dg.close()
