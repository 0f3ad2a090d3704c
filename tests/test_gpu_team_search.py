"""The team kernel (a CTA per query: row warps and a queue warp) and the merge
of small accepted batches, bit for bit against the oracle at the sizes where
they can go wrong: row widths on both sides of one register block, queues
around the 32-entry chunks, tables that spill, compact queues that rerun, rows
with and without 64 ids."""
import numpy as np
import pytest

from artea_b200.graph import CompactHierarchicalGraph
from artea_b200.router import DeviceIndex, GpuRouter
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF


def _graph(base, deg, seed, upper=True):
    """Level 0: ragged rows (0 to deg distinct ids, near ones and random ones); a few vertices on level 1."""
    rng = np.random.default_rng(seed)
    n = base.shape[0]
    d = (base ** 2).sum(1)[None, :] - 2.0 * base @ base.T
    np.fill_diagonal(d, np.inf)
    near = np.argsort(d, axis=1, kind="stable")[:, : deg // 2]
    up = np.sort(rng.choice(n, max(2, n // 50), replace=False)) if upper else np.zeros(0, int)
    highest = np.zeros(n, int)
    highest[up] = 1
    rows = []
    for v in range(n):
        far = rng.choice(n, deg, replace=False)
        ids = [int(x) for x in dict.fromkeys(np.concatenate([near[v], far]).tolist()) if x != v]
        level = [ids[: deg if v % 3 else int(rng.integers(0, deg + 1))]]
        if highest[v]:
            level.append([int(x) for x in rng.choice(up, min(len(up), 12), replace=False) if x != v])
        rows.append(level)
    entry = int(up[0]) if upper else 0
    return CompactHierarchicalGraph.from_rows(n, highest, rows, entry, bl_max_nbr_size=64)


def _data(n, dim, seed, levels=4):
    """Small whole numbers: distances tie often, and every sum is exact."""
    rng = np.random.default_rng(seed)
    return rng.integers(0, levels, (n, dim)).astype(np.float32)


@pytest.fixture(scope="module", params=[(16, 64), (128, 40), (144, 64), (960, 33)], ids=lambda p: f"dim{p[0]}-deg{p[1]}")
def case(request):
    dim, deg = request.param
    base = _data(1500, dim, dim)
    g = _graph(base, deg, dim)
    idx = DeviceIndex(g, base)
    yield g, base, _data(70, dim, dim + 1), idx
    idx.close()


@pytest.mark.parametrize("wpq", [1, 2, 4])
@pytest.mark.parametrize("queue", [1, 2, 31, 32, 33, 64, 97, 300])
def test_words_and_counters(case, wpq, queue):
    g, base, q, idx = case
    topk = min(queue, 50)
    ref, st = orc.batch_query(g, base, q, topk, queue, metric=0, stats=True)
    r = GpuRouter(idx, 0, topk, queue, warps_per_query=wpq, visited_hash_bits=8, schedule="persistent")
    out, got = r.batch_query(q, stats=True)
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(got[:, :7], st[:, :7])
    r.close()


@pytest.mark.parametrize("wpq", [2, 4])
@pytest.mark.parametrize("bits,slack", [(NONE, NONE), (6, NONE), (6, 1), (9, 64)])
def test_tables_that_spill_and_compact_queues(case, wpq, bits, slack):
    g, base, q, idx = case
    ref = orc.batch_query(g, base, q, 40, 150, metric=0)
    r = GpuRouter(idx, 0, 40, 150, warps_per_query=wpq, visited_hash_bits=bits, queue_slack=slack,
                  schedule="persistent")
    for _ in range(2):   # the visited set is left clear
        np.testing.assert_array_equal(r.batch_query(q), ref)
    r.close()


@pytest.mark.parametrize("wpq", [2, 4])
@pytest.mark.parametrize("metric", [1, 2, 3])
@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_metrics_and_modes(case, wpq, metric, mode):
    g, base, q, idx = case
    kw = dict(mode=mode, visited_hash_bits=9, schedule="persistent")
    if mode == "exact":
        ref = orc.batch_query(g, base, q, 30, 80, metric=metric)
    else:
        one = GpuRouter(idx, metric, 30, 80, warps_per_query=1, **kw)   # the same fold, one warp
        ref = one.batch_query(q)
        one.close()
    r = GpuRouter(idx, metric, 30, 80, warps_per_query=wpq, **kw)
    np.testing.assert_array_equal(r.batch_query(q), ref)
    np.testing.assert_array_equal(r.batch_query(q[:1]), ref[:1])
    r.close()


@pytest.mark.parametrize("wpq", [2, 4])
def test_per_query_sizes_level0_only_and_flat_graphs(case, wpq):
    g, base, q, idx = case
    rng = np.random.default_rng(5)
    queue = rng.choice([1, 7, 64, 200], q.shape[0]).astype(np.uint32)
    topk = np.minimum(queue, rng.choice([1, 5, 60], q.shape[0])).astype(np.uint32)
    kw = dict(warps_per_query=wpq, visited_hash_bits=8, schedule="persistent")
    r = GpuRouter(idx, 0, 60, 200, **kw)
    np.testing.assert_array_equal(r.batch_query(q, topk=topk, queue=queue, k_stride=60),
                                  orc.batch_query(g, base, q, topk, queue, metric=0, k_stride=60))
    np.testing.assert_array_equal(r.batch_query(q, l0_only=True),
                                  orc.batch_query(g, base, q, 60, 200, metric=0, l0_only=True))
    r.close()
    flat = _graph(base[:300], 20, 3, upper=False)
    fidx = DeviceIndex(flat, base[:300])
    r = GpuRouter(fidx, 0, 20, 400, **kw)   # a queue longer than the graph
    np.testing.assert_array_equal(r.batch_query(q), orc.batch_query(flat, base[:300], q, 20, 400, metric=0))
    r.close()
    fidx.close()
