"""Brute force where the tensor-core filter's bounds do not hold or its lists do
not fit, and calls that must not depend on it: the words are the oracle's."""
import threading

import numpy as np
import pytest

from artea_b200._native import ArteaGpuError
from artea_b200.router import DeviceIndex, vectors_only_graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _words(base, queries, k, metric):
    ids, d = orc.bruteforce(base, queries, k, metric=metric)
    return (d.view(np.uint32).astype(np.uint64) << np.uint64(32)) | ids.astype(np.uint64)


def _normal(n, dim, seed):
    return np.random.default_rng(seed).standard_normal((n, dim)).astype(np.float32)


@pytest.mark.parametrize("metric", [0, 1, 2, 3])
@pytest.mark.parametrize("exponent", [-9, -15, -17, -19, -21, -23])
def test_queries_of_small_norm(metric, exponent):
    """Squares of the elements underflow FP32 below about 1e-19."""
    base, q = _normal(9000, 64, 1), _normal(20, 64, 2)
    q *= np.float32(10.0 ** exponent)
    q[::5] *= np.float32(1e-2)
    idx = DeviceIndex(vectors_only_graph(), base)
    np.testing.assert_array_equal(idx.bruteforce(q, 12, metric), _words(base, q, 12, metric))
    idx.close()


def test_dot_query_whose_norm_underflows():
    """The nearest row is the one whose rounding to FP16 loses the most."""
    base = np.full((9000, 128), 0.5, np.float32)
    base[:2590:259] = 1.0 + 0.51 * 2.0 ** -10   # ten rows in ten tiles of 256
    base[5000, 0::2] = 1.0 + 1.49 * 2.0 ** -10
    base[5000, 1::2] = 1.0 + 0.49 * 2.0 ** -10
    q = np.full((4, 128), 2.6e-23, np.float32)
    q[:, 0] = 3e-23
    idx = DeviceIndex(vectors_only_graph(), base)
    got = idx.bruteforce(q, 10, 3)
    assert (got[:, 0] & np.uint64(0xFFFFFFFF) == 5000).all()
    np.testing.assert_array_equal(got, _words(base, q, 10, 3))
    idx.close()


@pytest.mark.parametrize("offset", [1, 2, 3])
@pytest.mark.parametrize("metric", [0, 2, 3])
def test_device_queries_at_any_float_offset(offset, metric):
    import torch
    base, q = _normal(9000, 80, 3), _normal(40, 80, 4)
    idx = DeviceIndex(vectors_only_graph(), base)
    flat = torch.zeros(q.size + 4, dtype=torch.float32, device="cuda")
    view = flat[offset:offset + q.size]
    view.copy_(torch.from_numpy(q.reshape(-1)))
    assert view.data_ptr() % 16 == 4 * offset
    want = _words(base, q, 10, metric)
    for nq in (2, 40, 3):   # few queries, the filter, few queries through the filter
        out = torch.zeros((nq, 10), dtype=torch.int64, device="cuda")
        idx.bruteforce_device(view, nq, 10, metric, out)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want[:nq])
    idx.close()


def test_calls_of_other_widths_at_the_same_time():
    """Each thread's calls on its own index and stream; widths, topk and row counts differ, so that
    the kernels want other amounts of shared memory in each."""
    import torch
    jobs = []
    for i, (n, dim, nq, k, metric) in enumerate([(9000, 64, 40, 10, 0), (8500, 960, 9, 100, 3), (9100, 400, 130, 1, 2),
                                                 (3000, 128, 20, 300, 1)]):
        base, q = _normal(n, dim, 10 + i), _normal(nq, dim, 20 + i)
        jobs.append((DeviceIndex(vectors_only_graph(), base), torch.from_numpy(q).cuda(), nq, k, metric,
                     _words(base, q, k, metric)))
    wrong = []

    def run(idx, dq, nq, k, metric, want):
        try:
            torch.cuda.set_device(0)
            s = torch.cuda.Stream()
            out = torch.zeros((nq, k), dtype=torch.int64, device="cuda")
            s.wait_stream(torch.cuda.current_stream())
            for _ in range(60):
                idx.bruteforce_device(dq, nq, k, metric, out, stream=s.cuda_stream)
                if not np.array_equal(out.cpu().numpy().view(np.uint64), want):
                    wrong.append((nq, k, metric))
        except Exception as e:   # a refused launch
            wrong.append(repr(e))

    threads = [threading.Thread(target=run, args=j) for j in jobs]
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not wrong, wrong[:4]
    for j in jobs:
        j[0].close()


def test_a_call_that_is_refused_leaves_the_workspace_to_the_next():
    """Waiting for a stream that is being captured is refused, in the middle of a call."""
    import torch
    from cuda.bindings import runtime as rt
    base, q = _normal(9000, 64, 5), _normal(30, 64, 6)
    idx = DeviceIndex(vectors_only_graph(), base)
    want = _words(base, q, 10, 0)
    dq = torch.from_numpy(q).cuda()
    out = torch.zeros((30, 10), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for nq in (30, 2):
        s = torch.cuda.Stream()
        assert rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0] == 0
        with pytest.raises(RuntimeError):
            idx.bruteforce_device(dq, nq, 10, 0, out, stream=s.cuda_stream)
        rt.cudaStreamEndCapture(s.cuda_stream)
        rt.cudaGetLastError()
        idx.bruteforce_device(dq, nq, 10, 0, out[:nq])
        np.testing.assert_array_equal(out[:nq].cpu().numpy().view(np.uint64), want[:nq])
    idx.close()


@pytest.mark.parametrize("nq", [2, 5])
@pytest.mark.parametrize("n,dim,topk", [(8300, 3200, 1024), (8300, 6752, 256)])
def test_tiles_above_the_scans_shared_memory_are_refused(n, dim, topk, nq):
    """8 queries' lists and rows in 227 KB: the last dims that fit are 3,152 at topk 1,024 and 6,224 at 256."""
    base, q = _normal(n, dim, 7), _normal(nq, dim, 8)
    idx = DeviceIndex(vectors_only_graph(), base)
    with pytest.raises(ArteaGpuError, match="EINVAL"):
        idx.bruteforce(q, topk, 0)
    idx.close()


@pytest.mark.parametrize("metric", [0, 1, 2, 3])
@pytest.mark.parametrize("n,nq", [(9000, 2), (9000, 24), (9000, 300), (40000, 13)])
def test_queries_whose_lists_overflow_are_scanned_together(n, nq, metric):
    """Half of the queries are nearest to one row that is there 6,000 times: more than a list holds."""
    rng = np.random.default_rng(n + nq)
    base = rng.integers(-8, 9, (n, 48)).astype(np.float32)
    base[100:6100] = 20.0
    q = rng.integers(-8, 9, (nq, 48)).astype(np.float32)
    q[::2] = 19.0 + rng.integers(0, 3, (len(q[::2]), 48))
    idx = DeviceIndex(vectors_only_graph(), base)
    np.testing.assert_array_equal(idx.bruteforce(q, 30, metric), _words(base, q, 30, metric))
    last = idx.last_bruteforce()
    assert last["scans"] == 1 and len(q[::2]) <= last["scanned"] < nq, last
    idx.close()


@pytest.mark.parametrize("metric", [0, 2, 3])
@pytest.mark.parametrize("nq", [4, 130])
def test_every_list_overflows(nq, metric):
    """All rows but 100 equal: a list is full after a few tiles, and the rest of them is not listed."""
    base, q = np.tile(_normal(1, 48, 13), (70000, 1)), _normal(nq, 48, 14)
    base[30000:30100] = _normal(100, 48, 15)
    q[2] = base[30050]
    idx = DeviceIndex(vectors_only_graph(), base)
    np.testing.assert_array_equal(idx.bruteforce(q, 20, metric), _words(base, q, 20, metric))
    assert idx.last_bruteforce()["scans"] == 1 and idx.last_bruteforce()["scanned"] >= nq - 1
    idx.close()


@pytest.mark.parametrize("metric", [0, 1, 3])
def test_one_large_query_does_not_send_the_others_to_the_scan(metric):
    base, q = _normal(20000, 64, 11), _normal(150, 64, 12)
    q[17] *= np.float32(1e12)
    idx = DeviceIndex(vectors_only_graph(), base)
    np.testing.assert_array_equal(idx.bruteforce(q, 10, metric), _words(base, q, 10, metric))
    assert idx.last_bruteforce()["scanned"] <= 1
    idx.close()


@pytest.mark.parametrize("metric", [0, 2, 3])
@pytest.mark.parametrize("nq", [3, 40])
def test_subset_with_repeated_ids(nq, metric):
    """An id comes as often as the subset holds it; the words are in order of (distance, id)."""
    rng = np.random.default_rng(16)
    base, q = _normal(12000, 96, 17), _normal(nq, 96, 18)
    sub = rng.permutation(12000)[:6000].astype(np.uint32)
    sub = rng.permutation(np.concatenate([sub, sub[:3000], sub[:500], sub[:100]]))
    rows = np.sort(sub)   # the oracle's ties: by position
    ids, d = orc.bruteforce(base[rows], q, 60, metric=metric)
    want = (d.view(np.uint32).astype(np.uint64) << np.uint64(32)) | rows[ids].astype(np.uint64)
    assert (want[:, 1:] == want[:, :-1]).any()
    idx = DeviceIndex(vectors_only_graph(), base)
    np.testing.assert_array_equal(idx.bruteforce(q, 60, metric, sub), want)
    idx.bruteforce(q, 60, metric)
    np.testing.assert_array_equal(idx.bruteforce(q, 60, metric, sub), want)
    idx.close()
