"""The end of a persistent launch with CTAs of four warps, where the warps without
a query become row warps of the last one: words and counters against the oracle
for batches that leave most warps idle, rows that the three row warps divide
unevenly, tables that spill, compact queues that rerun, one and two passes a slice."""
import numpy as np
import pytest

from artea_b200.graph import CompactHierarchicalGraph
from artea_b200.router import DeviceIndex, GpuRouter
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF


def _graph(n, deg, seed):
    rng = np.random.default_rng(seed)
    rows = []
    for v in range(n):
        ids = [int(x) for x in rng.choice(n, deg, replace=False) if x != v]
        rows.append([ids[: deg if v % 3 else int(rng.integers(0, deg + 1))]])
    return CompactHierarchicalGraph.from_rows(n, np.zeros(n, int), rows, 0, bl_max_nbr_size=64)


@pytest.fixture(scope="module", params=[(16, 64, 0), (128, 23, 0), (96, 45, 2)], ids=lambda p: f"dim{p[0]}-deg{p[1]}")
def case(request):
    dim, deg, metric = request.param
    rng = np.random.default_rng(dim)
    base = rng.integers(0, 4, (1200, dim)).astype(np.float32)
    base[:, 0] += 1.0   # no zero vector (cosine)
    queries = rng.integers(0, 4, (90, dim)).astype(np.float32) + 1.0
    g = _graph(1200, deg, deg)
    idx = DeviceIndex(g, base)
    yield g, base, queries, metric, idx
    idx.close()


@pytest.mark.parametrize("budget", [96, 128])
@pytest.mark.parametrize("bits,slack,queue", [(9, NONE, 1), (9, NONE, 33), (9, NONE, 200), (6, NONE, 150), (NONE, NONE, 90),
                                              (8, 1, 120)])
def test_words_and_counters(case, budget, bits, slack, queue):
    g, base, q, metric, idx = case
    topk = min(queue, 50)
    ref, st = orc.batch_query(g, base, q, topk, queue, metric=metric, stats=True)
    r = GpuRouter(idx, metric, topk, queue, warps_per_cta=4, register_budget=budget, visited_hash_bits=bits,
                  queue_slack=slack, stage_rows=NONE, pipeline=1, schedule="persistent")
    for nq in (1, 2, 7, 90):
        out, got = r.batch_query(q[:nq], stats=True)
        np.testing.assert_array_equal(out, ref[:nq])
        np.testing.assert_array_equal(got[:, :7], st[:nq, :7])
    r.close()
