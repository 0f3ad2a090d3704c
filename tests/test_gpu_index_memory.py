"""The copies an index keeps beside its vectors and CSR (level-0 rows at a fixed
stride, FP16 rows of brute force): counted, given back, and not made where the
device has no room for them."""
import numpy as np
import pytest

from artea_b200._native import ArteaGpuError
from artea_b200.router import DeviceIndex, GpuRouter, vectors_only_graph
from oracle import oracle as orc
from test_gpu_team_search import _data, _graph

pytestmark = pytest.mark.gpu

GB = 1 << 30


def _fill(leave):
    """Takes the device's memory but `leave` bytes."""
    import torch
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(max(0, free - leave), dtype=torch.uint8, device="cuda")


def _search(idx, g, base, q):
    ref, st = orc.batch_query(g, base, q, 20, 60, metric=0, stats=True)
    for kw in (dict(), dict(warps_per_query=1), dict(warps_per_query=2), dict(pipeline=1), dict(schedule="plain")):
        r = GpuRouter(idx, 0, 20, 60, **kw)
        out, got = r.batch_query(q, stats=True)
        np.testing.assert_array_equal(out, ref)
        np.testing.assert_array_equal(got[:, :7], st[:, :7])
        r.close()


def test_copies_are_counted_and_given_back():
    base, q = _data(9000, 80, 1, 50), _data(40, 80, 2, 50)
    g = _graph(base, 24, 3)
    idx = DeviceIndex(g, base)
    whole = idx.nbytes()
    want = idx.bruteforce(q, 10, 0)
    assert idx.nbytes() == whole + 9000 * 128 * 2 and idx.last_bruteforce()["scanned"] == 0
    r = GpuRouter(idx, 0, 20, 60)
    with pytest.raises(ArteaGpuError, match="EINVAL"):
        idx.lean()
    r.close()
    idx.lean()
    assert idx.nbytes() == whole - 9000 * 256
    np.testing.assert_array_equal(idx.bruteforce(q, 10, 0), want)
    assert idx.last_bruteforce()["scanned"] == 40 and idx.nbytes() == whole - 9000 * 256
    _search(idx, g, base, q)
    idx.close()


def test_no_fixed_stride_rows_on_a_full_device():
    import torch
    base, q = _data(1500, 48, 4), _data(20, 48, 5)
    g = _graph(base, 24, 6)
    other = DeviceIndex(g, base)
    _search(other, g, base, q)   # the kernels are loaded
    whole = other.nbytes()
    other.close()
    fill = _fill(GB // 2)
    try:
        idx = DeviceIndex(g, base)
        assert idx.nbytes() == whole - 1500 * 256
        _search(idx, g, base, q)
        idx.close()
    finally:
        del fill
        torch.cuda.empty_cache()


def test_rounded_rows_are_made_once_there_is_room():
    import torch
    base = np.random.default_rng(7).standard_normal((1_000_000, 64), dtype=np.float32)
    q = np.random.default_rng(8).standard_normal((30, 64), dtype=np.float32)
    idx = DeviceIndex(vectors_only_graph(), base)
    before = idx.nbytes()
    fill = _fill(GB // 2)
    try:
        scanned = idx.bruteforce(q, 10, 0)
        assert idx.last_bruteforce()["scanned"] == 30 and idx.nbytes() == before
    finally:
        del fill
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(idx.bruteforce(q, 10, 0), scanned)
    assert idx.last_bruteforce()["scanned"] == 0 and idx.nbytes() == before + 1_000_000 * 128
    idx.close()


def test_saved_picks_stay_with_the_rows_they_were_timed_with(tmp_path, monkeypatch):
    """Teams of 2, 4 and 8 row warps exist for fixed-stride rows alone, teams of 1 and 3 without them alone;
    two indexes that differ in nothing else share a tuning file."""
    path = tmp_path / "tuning.txt"
    monkeypatch.setenv("ARTEA_TUNING_CACHE", str(path))
    base, q = _data(1500, 48, 4), _data(20, 48, 5)
    g = _graph(base, 24, 6)
    ref = orc.batch_query(g, base, q, 20, 60, metric=0)
    whole, lean = DeviceIndex(g, base), DeviceIndex(g, base)
    lean.lean()

    def run(idx):
        r = GpuRouter(idx, 0, 20, 60, schedule="persistent")
        np.testing.assert_array_equal(r.batch_query(q), ref)
        t = r.tuning()
        r.close()
        return t

    for first, second, teams in ((whole, lean, (2, 4, 8)), (lean, whole, (1, 3))):
        path.write_text("")
        run(first)
        key = path.read_text().split()[0]
        for team in teams:
            path.write_text(f"{key} 1 8 2 0 0 0 {team} 0\n")   # the pick: this team
            assert run(first)["warps_per_cta"] == team
            run(second)
            assert len({line.split()[0] for line in path.read_text().splitlines()}) == 2
    whole.close()
    lean.close()


def test_a_router_closed_after_its_index_leaves_the_next_index_alone():
    """The next index mostly takes the memory of the one destroyed before it; its count of routers stays 0."""
    base = _data(300, 16, 1)
    g = _graph(base, 24, 2)
    for _ in range(8):
        idx = DeviceIndex(g, base)
        routers = [GpuRouter(idx, 0, 5, 20) for _ in range(3)]
        idx.close()
        following = DeviceIndex(g, base)
        for r in routers:
            r.close()
        following.lean()   # refused while a router is alive on it
        following.close()
