"""The tensor-core filter in front of exact brute force: the words must be the
FP32 scan's on every input, at the edges of its tiles (128 queries, 256 rows, 64
elements) and where its bounds are loose or do not hold (ties, rows of very
different norms, values that are not finite, subsets with repeats)."""
import numpy as np
import pytest

from artea_b200.router import DeviceIndex, vectors_only_graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _rows(n, dim, seed, kind="normal"):
    rng = np.random.default_rng(seed)
    if kind == "whole":
        return rng.integers(0, 3, (n, dim)).astype(np.float32)
    if kind == "clusters":   # one after the other, so that near rows share tiles
        c = rng.standard_normal((n // 500 + 1, dim))
        return (np.repeat(c, 500, axis=0)[:n] + 0.1 * rng.standard_normal((n, dim))).astype(np.float32)
    return rng.standard_normal((n, dim)).astype(np.float32)


def _words(base, queries, k, metric, subset=None):
    rows = np.arange(len(base)) if subset is None else np.sort(subset)   # the oracle's ties: by position
    ids, d = orc.bruteforce(base[rows], queries, k, metric=metric)
    return (d.view(np.uint32).astype(np.uint64) << np.uint64(32)) | rows[ids].astype(np.uint64)


def _check(base, queries, k, metric, subset=None):
    idx = DeviceIndex(vectors_only_graph(), base)
    want = _words(base, queries, k, metric, subset)
    # Few queries while the index holds no rounded rows: FP32 throughout.
    np.testing.assert_array_equal(idx.bruteforce(queries[:2], k, metric, subset), want[:2])
    np.testing.assert_array_equal(idx.bruteforce(queries, k, metric, subset), want)
    # Few queries, on the rounded rows that the index holds by now.
    np.testing.assert_array_equal(idx.bruteforce(queries[:3], k, metric, subset), want[:3])
    idx.close()


@pytest.mark.parametrize("n,nq,dim,k", [(8192, 16, 16, 1), (8193, 127, 64, 10), (8447, 128, 80, 17), (9000, 129, 128, 100),
                                        (20000, 300, 96, 64), (8448, 40, 400, 5), (8200, 33, 960, 1024)])
@pytest.mark.parametrize("metric", [0, 1, 2, 3])
def test_edges(n, nq, dim, k, metric):
    _check(_rows(n, dim, n), _rows(nq, dim, nq + 1), k, metric)


@pytest.mark.parametrize("metric", [0, 1, 2, 3])
@pytest.mark.parametrize("kind", ["whole", "clusters"])
def test_ties_and_neighbours_in_one_tile(kind, metric):
    base = _rows(12000, 48, 5, kind)
    base[100:160] = base[99]      # repeated rows
    base[7] = 0.0                 # a zero row
    q = np.concatenate([base[rng] for rng in (slice(90, 110), slice(0, 12), slice(11990, 12000))])
    q[3] = 0.0                    # a zero query
    _check(base, q, 100, metric)


@pytest.mark.parametrize("metric", [0, 2, 3])
@pytest.mark.parametrize("what", ["inf", "nan", "huge", "tiny", "spread"])
def test_norms_outside_the_bounds(what, metric):
    base, q = _rows(9000, 32, 1), _rows(20, 32, 2)
    if what == "huge":
        base *= np.float32(1e17)
    elif what == "tiny":
        base[::2] *= np.float32(1e-12)
    elif what == "spread":
        base *= np.float32(10.0) ** np.random.default_rng(3).integers(-6, 6, (9000, 1)).astype(np.float32)
        q[::3] *= np.float32(1e5)
    else:
        q[4, 5] = np.inf if what == "inf" else np.nan
        q[9, 0] = -np.inf if what == "inf" else np.nan
    idx = DeviceIndex(vectors_only_graph(), base)
    got = idx.bruteforce(q, 20, metric)
    # Reference: FP32 throughout (few queries on an index without rounded rows).
    other = DeviceIndex(vectors_only_graph(), base)
    want = np.concatenate([other.bruteforce(q[i:i + 2], 20, metric) for i in range(0, 20, 2)])
    np.testing.assert_array_equal(got, want)
    idx.close()
    other.close()


@pytest.mark.parametrize("metric", [0, 2])
def test_subset(metric):
    rng = np.random.default_rng(9)
    base, q = _rows(30000, 96, 4, "clusters"), _rows(50, 96, 6, "clusters")
    sub = rng.permutation(30000)[:8300].astype(np.uint32)
    _check(base, q, 10, metric, sub)


def test_many_queries_and_device_buffers():
    import torch
    base, q = _rows(10000, 64, 7), _rows(2200, 64, 8)   # more than one batch of queries
    idx = DeviceIndex(vectors_only_graph(), base)
    dq = torch.from_numpy(q).cuda()
    out = torch.zeros((2200, 10), dtype=torch.int64, device="cuda")
    idx.bruteforce_device(dq, 2200, 10, 0, out)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), _words(base, q, 10, 0))
    idx.close()
