"""The autotuner's candidates: the plain path's geometry is the first of them (or, where smaller tables
hold every rank, the same CTA count with a smaller table, which runs the same), and every candidate's
CTAs are resident together on an SM."""
import os
import re
import subprocess
import sys
import threading

import pytest

import oracle
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200._ffi import PBError
from parbutterfly_b200.graph import BipartiteGraph

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
from parbutterfly_b200 import butterflies as pb
from parbutterfly_b200._ffi import PBError
from parbutterfly_b200.graph import BipartiteGraph
with pb.Context(0) as ctx:
    dg = ctx.upload(BipartiteGraph.rmat(SCALE, SCALE - 2, 60000, 0.55, 0.15, 0.15, 0.15, 73))
    plain = pb.count(dg, "HASH", "ADEG")
    st = ctx.stats()
    print("plain", st["count_smem_bytes"], st["count_blocks_per_sm"], st["count_small_w"])
    assert (pb.count(dg, "HASH", "ADEG", autotune=True) == plain).all()
    st = ctx.stats()
    print("tuned", st["count_smem_bytes"], st["count_blocks_per_sm"], st["count_small_w"])
"""


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [12, 15])  # 5120 and 40960 vertices; 48 KiB hold the counters of 20,000
def test_plain_geometry_is_a_candidate(scale):
    r = subprocess.run([sys.executable, "-c", SCRIPT.replace("SCALE", str(scale))], cwd=ROOT,
                       env=dict(os.environ, PB_TRACE="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    said = {ln.split()[0]: tuple(map(int, ln.split()[1:])) for ln in r.stdout.splitlines()}
    tried = [tuple(map(int, t)) for t in re.findall(r"autotune (\d+) bytes x (\d+) CTAs, warp (\d+)", r.stderr)]
    assert said["tuned"] in tried and len(set(tried)) == len(tried)
    if scale == 15:
        assert tried[0] == said["plain"]
    else:
        assert tried[0][0] < said["plain"][0] and tried[0][1:] == said["plain"][1:]
    for smem, ctas, _ in tried:
        assert ctas * (smem + 1024) <= 228 * 1024 and ctas * 512 * 40 <= 65536  # 40 registers a thread


@pytest.mark.gpu
def test_threads_with_different_geometries():
    """Two threads tune (tables of up to 200 KiB a CTA, tuned anew on every context), two count with the
    plain geometry."""
    gs = [BipartiteGraph.rmat(12, 10, 60000 + 10 * k, 0.55, 0.15, 0.15, 0.15, 80 + k) for k in range(100)]
    want = [oracle.count(g, "TOTAL", "ADEG")[0] for g in gs]
    failures, tuning = [], [2]

    def work(tune):
        try:
            for _ in range(8 if tune else 1000):
                with pb.Context(0) as ctx:
                    for g, w in zip(gs, want):
                        dg = ctx.upload(g)
                        try:
                            if pb.count_total(dg, "HASH", "ADEG", autotune=tune) != w:
                                failures.append("totals differ")
                        except PBError as e:
                            failures.append(str(e))
                        dg.close()
                if tuning[0] == 0:
                    break
        finally:
            if tune:
                tuning[0] -= 1

    threads = [threading.Thread(target=work, args=(t,)) for t in (True, True, False, False)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failures == []
