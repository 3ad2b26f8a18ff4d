"""Timed cases of the counting and peeling entry points.

Each case is one call (or the few calls) that a program makes on a graph it already holds:
`prepare` builds the seeded graph on the GPU and whatever that program keeps (the context, the
uploaded graph, output buffers, the counts a peel starts from); `run` is one pass through the
public entry points.  Graph families and sizes follow the repository's own workloads: uniform
and Zipf endpoints, bipartite R-MAT (.55, .15, .15, .15), power-law U degrees, and batches of
uneven graphs.
"""
import math
import random

import numpy as np
import torch

from parbutterfly_b200 import butterflies as pb

RMAT = (0.55, 0.15, 0.15, 0.15)


def listed():
    return [
        # A call on a graph so small that only launches and synchronisation count.
        {"name": "total_tiny", "path": "count", "per": "TOTAL", "count_type": "BATCHS", "rank_type": "ADEG",
         "graph": "uniform", "nv": 300, "nu": 180, "m": 1777},
        # The small plain-method workload: 4096 x 4096, 131072 uniform edges, per vertex.
        {"name": "vert_uniform_4096", "path": "count", "per": "VERT", "count_type": "BATCHS", "rank_type": "ADEG",
         "graph": "uniform", "nv": 4096, "nu": 4096, "m": 131072},
        # Per-edge counts of an ordinary skewed graph, as wing peeling needs them.
        {"name": "edge_rmat18", "path": "count", "per": "EDGE", "count_type": "HASH", "rank_type": "ACOCORE",
         "graph": "rmat", "nv": 1 << 14, "nu": 1 << 12, "m": 1 << 18},
        # The benchmark graph's per-edge counts, kept on the device for the peel that follows.
        {"name": "edge_rmat24", "path": "count", "per": "EDGE", "count_type": "HASH", "rank_type": "ACOCORE",
         "graph": "rmat", "nv": 1 << 20, "nu": 1 << 18, "m": 1 << 24, "device_out": True},
        # Per-vertex counts with power-law degrees (the 1e7-edge member of that workload).
        {"name": "vert_powerlaw_10m", "path": "count", "per": "VERT", "count_type": "BATCHS", "rank_type": "ADEG",
         "graph": "powerlaw", "nv": 100_000, "nu": 1_000_000, "m": 10_000_000, "device_out": True},
        # The sort-based aggregation on skewed endpoints, ragged sizes.
        {"name": "vert_sort_zipf", "path": "count", "per": "VERT", "count_type": "SORT", "rank_type": "DEG",
         "graph": "zipf", "nv": 30_011, "nu": 20_021, "m": 300_007},
        # The histogram aggregation per edge under the exact co-core order.
        {"name": "edge_hist_cocore", "path": "count", "per": "EDGE", "count_type": "HIST", "rank_type": "COCORE",
         "graph": "uniform", "nv": 50_021, "nu": 33_013, "m": 1_000_003},
        # A program that reads a graph file's text and counts it once, as the command line does.
        {"name": "load_text", "path": "load", "per": "VERT", "count_type": "SERIAL", "rank_type": "SIDE",
         "graph": "uniform", "nv": 20_011, "nu": 30_029, "m": 400_009},
        # Tip numbers, the exact rounds one after another.
        {"name": "tip_rmat20", "path": "tip", "parts": 0, "graph": "rmat", "nv": 1 << 16, "nu": 1 << 14, "m": 1 << 20},
        # Tip numbers of a larger graph with the rounds batched.
        {"name": "tip_parts_rmat22", "path": "tip", "parts": 296, "graph": "rmat", "nv": 1 << 18, "nu": 1 << 16,
         "m": 1 << 22},
        # Wing numbers of an ordinary graph (the size compared with the CPU implementation).
        {"name": "wing_rmat18", "path": "wing", "graph": "rmat", "nv": 1 << 14, "nu": 1 << 12, "m": 1 << 18},
        # Many uneven graphs counted and peeled together.
        {"name": "batch_64", "path": "batch", "k": 64, "sizes": 4000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rmat_dims(m):
    # 2^20 x 2^18 at 2^24 edges, the same density at every size.
    lv = max(6, round(math.log2(m)) - 4)
    return 1 << lv, 1 << max(5, lv - 2)


def draw(rng):
    """One more case of the same ranges (no name)."""
    kind = rng.choice(["small", "small", "fused", "fused", "materialised", "load", "tip", "parts", "wing", "batch"])
    per = rng.choice(["VERT", "EDGE", "TOTAL"])
    rank = rng.choice(["SIDE", "DEG", "ADEG", "COCORE", "ACOCORE"])
    fused = rng.choice(["HASH", "BATCHS", "BATCHWA", "SERIAL"])
    if kind == "small":
        m = _log_int(rng, 1_000, 130_000)
        nv, nu = _log_int(rng, 100, 5_000), _log_int(rng, 100, 5_000)
        return {"path": "count", "per": per, "count_type": fused, "rank_type": rank,
                "graph": rng.choice(["uniform", "zipf"]), "nv": nv, "nu": nu, "m": min(m, nv * nu // 4)}
    if kind == "fused":
        m = _log_int(rng, 150_000, 9_000_000)
        if rng.random() < 0.5:
            nv, nu = _rmat_dims(m)
            return {"path": "count", "per": per, "count_type": fused, "rank_type": rank, "graph": "rmat", "nv": nv,
                    "nu": nu, "m": m, "device_out": rng.random() < 0.5}
        return {"path": "count", "per": per, "count_type": fused, "rank_type": rank, "graph": "powerlaw",
                "nv": max(1000, m // 100), "nu": m // 10, "m": m, "device_out": rng.random() < 0.5}
    if kind == "materialised":
        m = _log_int(rng, 10_000, 1_000_000)
        graph = rng.choice(["uniform", "zipf"])
        if graph == "zipf":
            m = min(m, 300_000)
        return {"path": "count", "per": per, "count_type": rng.choice(["SORT", "ASORT", "HIST", "AHIST"]),
                "rank_type": rank, "graph": graph, "nv": m // rng.randint(8, 24), "nu": m // rng.randint(8, 24), "m": m}
    if kind == "load":
        m = _log_int(rng, 10_000, 400_000)
        return {"path": "load", "per": "VERT", "count_type": fused, "rank_type": rng.choice(["SIDE", "DEG", "ADEG"]),
                "graph": "uniform", "nv": m // rng.randint(8, 24), "nu": m // rng.randint(8, 24), "m": m}
    if kind == "tip":
        m = _log_int(rng, 16_000, 1_000_000)
        nv, nu = _rmat_dims(m)
        return {"path": "tip", "parts": 0, "graph": "rmat", "nv": nv, "nu": nu, "m": m}
    if kind == "parts":
        m = _log_int(rng, 500_000, 4_000_000)
        nv, nu = _rmat_dims(m)
        return {"path": "tip", "parts": rng.choice([148, 296, 592]), "graph": "rmat", "nv": nv, "nu": nu, "m": m}
    if kind == "wing":
        m = _log_int(rng, 4_000, 250_000)
        nv, nu = _rmat_dims(m)
        return {"path": "wing", "graph": "rmat", "nv": nv, "nu": nu, "m": m}
    return {"path": "batch", "k": rng.randint(4, 56), "sizes": rng.randint(1, 1 << 20)}


# ---- graphs ----------------------------------------------------------------------------------
def _pairs(case, n, gen):
    """n endpoint pairs (v, u) of the case's family, duplicates included."""
    dev, nv, nu = "cuda", case["nv"], case["nu"]

    def unit():
        return torch.rand(n, generator=gen, device=dev, dtype=torch.float64)

    def below(k):
        return torch.randint(0, k, (n,), generator=gen, device=dev, dtype=torch.int64)

    if case["graph"] == "uniform":
        return below(nv), below(nu)
    if case["graph"] == "zipf":  # exponent 1.5 on both sides (the batch workload's skewed half)
        def zipf(k):
            cdf = torch.cumsum(torch.arange(1, k + 1, device=dev, dtype=torch.float64) ** -1.5, 0)
            return torch.searchsorted(cdf / cdf[-1], unit()).clamp_(max=k - 1)
        return zipf(nv), zipf(nu)
    if case["graph"] == "powerlaw":  # U degrees ~ k^-2, capped at |V| by the distinctness of pairs
        w = 1.0 / (1.0 - (torch.arange(nu, device=dev, dtype=torch.float64) + 0.5) / nu)
        w = w[torch.randperm(nu, generator=gen, device=dev)]
        cdf = torch.cumsum(w.clamp(max=float(w.sum()) * nv / case["m"]), 0)
        return below(nv), torch.searchsorted(cdf / cdf[-1], unit()).clamp_(max=nu - 1)
    a, b, c, _ = RMAT
    lv, lu = nv.bit_length() - 1, nu.bit_length() - 1
    v = torch.zeros(n, dtype=torch.int64, device=dev)
    u = torch.zeros(n, dtype=torch.int64, device=dev)
    for level in range(max(lv, lu)):
        r = unit()
        if level < lv:
            v = 2 * v + (r >= a + b)
        if level < lu:
            u = 2 * u + (((r >= a) & (r < a + b)) | (r >= a + b + c))
    return v, u


def _edges(case, gen):
    """Exactly case["m"] distinct edges as sorted keys v * nu + u."""
    nv, nu, m = case["nv"], case["nu"], case["m"]
    keys = torch.zeros(0, dtype=torch.int64, device="cuda")
    for attempt in range(12):
        want = m - keys.numel()
        if want <= 0:
            break
        # Saturated skewed graphs top up with uniform pairs after a few tries.
        src = case if attempt < 6 else dict(case, graph="uniform")
        v, u = _pairs(src, want + want // 8 + 64, gen)
        keys = torch.unique(torch.cat([keys, v * nu + u]))
    if keys.numel() > m:
        keep = torch.randperm(keys.numel(), generator=gen, device="cuda")[:m]
        keys = torch.sort(keys[keep])[0]
    return keys


def _offsets(ids, n):
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(ids, minlength=n), 0)
    return off.to(torch.int32)


def _csr(case, gen):
    """(nv, nu, offV, edgV, offU, edgU): both CSR sides on the GPU, 32-bit ids."""
    nv, nu = case["nv"], case["nu"]
    keys = _edges(case, gen)
    v, u = keys // nu, keys % nu
    turned = torch.sort(u * nv + v)[0]
    return (nv, nu, _offsets(v, nv), u.to(torch.int32), _offsets(u, nu), (turned % nv).to(torch.int32))


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _upload(ctx, arrays):
    torch.cuda.synchronize()  # the context has a stream of its own
    return pb.DeviceGraph(ctx, device_arrays=arrays)


def _batch_members(case):
    """Sizes of a batch's graphs: sides log-uniform in [64, 65536], 4 to 64 edges per vertex."""
    rng = random.Random(case["sizes"])
    for _ in range(case["k"]):
        nu, nv = _log_int(rng, 64, 65536), _log_int(rng, 64, 65536)
        m = int(round(math.exp(rng.uniform(math.log(4), math.log(64))) * min(nu, nv)))
        yield {"graph": rng.choice(["uniform", "zipf"]), "nv": nv, "nu": nu, "m": min(m, nv * nu // 2)}


def _text(arrays):
    """The graph as AdjacencyHypergraph text."""
    nv, nu, off_v, edg_v, off_u, edg_u = arrays
    m = edg_v.numel()
    nums = [np.array([nv, m, nu, m])] + [t.cpu().numpy() for t in (off_v[:-1], edg_v, off_u[:-1], edg_u)]
    return ("AdjacencyHypergraph\n" + "\n".join(map(str, np.concatenate(nums).tolist())) + "\n").encode()


# ---- the passes ------------------------------------------------------------------------------
def prepare(case, seed):
    gen = _generator(seed)
    ctx = pb.Context(0)
    state = {"case": case, "ctx": ctx}
    if case["path"] == "batch":
        state["graphs"] = [_upload(ctx, _csr(member, gen)) for member in _batch_members(case)]
        return state
    arrays = _csr(case, gen)
    if case["path"] == "load":
        state["text"] = _text(arrays)
        return state
    dg = state["graph"] = _upload(ctx, arrays)
    use_v, _ = pb.cmp_wedge_counts(dg)
    side = dg.nu if use_v else dg.nv

    def buffer(n):
        return torch.zeros(n, dtype=torch.int64, device="cuda")

    if case["path"] == "count" and case.get("device_out") and case["per"] != "TOTAL":
        state["out"] = buffer(dg.m if case["per"] == "EDGE" else side)
    if case["path"] == "tip":
        state["counts"], state["out"] = buffer(side), buffer(side)
        torch.cuda.synchronize()
        pb.count(dg, "BATCHS", "ADEG", out=state["counts"])
    if case["path"] == "wing":
        state["counts"], state["out"] = buffer(dg.m), buffer(dg.m)
        torch.cuda.synchronize()
        pb.count_e(dg, "HASH", "ACOCORE", out=state["counts"])
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["path"] == "count":
        dg, how = state["graph"], (case["count_type"], case["rank_type"])
        if case["per"] == "TOTAL":
            return pb.count_total(dg, *how)
        return (pb.count_e if case["per"] == "EDGE" else pb.count)(dg, *how, out=state.get("out"))
    if case["path"] == "load":
        dg = pb.graph_from_text(state["ctx"], state["text"])
        counts = pb.count(dg, case["count_type"], case["rank_type"])
        dg.close()
        return counts
    if case["path"] == "tip":
        return pb.peel(state["graph"], state["counts"], out=state["out"], peel_parts=case["parts"])
    if case["path"] == "wing":
        return pb.peel_e(state["graph"], state["counts"], out=state["out"])
    counts = pb.count_batch(state["graphs"], "BATCHS", "ADEG")
    tips = pb.peel_batch(state["graphs"], counts)
    return {"counts": np.concatenate(counts), "tips": np.concatenate(tips)}


def work(case):
    """Bytes: both CSR sides (the text, when loading) read once, the result written once and, for
    a peel, the counts it starts from read once.  The wedges a pass walks depend on the graph and
    are not in a closed form, so no operations are claimed."""
    if case["path"] == "batch":
        return {"bytes": sum(4 * (g["nv"] + g["nu"] + 2 + 2 * g["m"]) + 16 * min(g["nv"], g["nu"])
                             for g in _batch_members(case)), "flops": 0}
    nv, nu, m = case["nv"], case["nu"], case["m"]
    graph = 4 * (nv + nu + 2 + 2 * m)
    if case["path"] == "load":
        graph = 6 * (nv + nu + 2 * m)  # five digits and a separator for most numbers
    items = {"VERT": min(nv, nu), "EDGE": m, "TOTAL": 1}[case.get("per", "EDGE" if case["path"] == "wing" else "VERT")]
    return {"bytes": graph + (8 if case["path"] in ("count", "load") else 16) * items, "flops": 0}


def exact(case, seed):
    """Counts from the dense adjacency matrix in 64 bits: W = A^T A holds the common neighbours of
    every pair of count-side vertices.  None for peels, batches and graphs too large to be dense."""
    if case["path"] not in ("count", "load") or case["nv"] * case["nu"] > 1 << 27:
        return None
    nv, nu, off_v, edg_v, _, _ = _csr(case, _generator(seed))
    deg = (off_v[1:] - off_v[:-1]).to(torch.int64)
    v = torch.repeat_interleave(torch.arange(nv, device="cuda"), deg)
    a = torch.zeros(nv, nu, dtype=torch.float64, device="cuda")
    a[v, edg_v.to(torch.int64)] = 1.0

    def wedges(degrees):  # the count side is chosen by 32-bit products, summed in 64 bits
        d = degrees.to(torch.int64)
        return int((((d * (d - 1)) & 0xFFFFFFFF) // 2).sum())

    if wedges(a.sum(1)) > wedges(a.sum(0)):
        a = a.t().contiguous()  # rows: centre side, columns: count side
    if a.shape[1] > 1 << 15:
        return None
    w = a.t() @ a
    if case["per"] == "EDGE":
        common = (a @ w)[a > 0]  # row-major: the order of the centre side's lists
        row, col = torch.nonzero(a, as_tuple=True)
        out = common - a.sum(0)[col] - a.sum(1)[row] + 1
        return out.round().to(torch.int64)
    w.fill_diagonal_(0.0)
    per_vertex = (w * (w - 1) / 2).sum(1).round().to(torch.int64)
    return int(per_vertex.sum()) // 2 if case["per"] == "TOTAL" else per_vertex
