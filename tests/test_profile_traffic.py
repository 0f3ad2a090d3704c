"""DRAM traffic from a committed ncu summary: only for the launch and the kernels it was captured with."""
import json

import pytest

import bench

TUNING = {"warps_per_cta": 4, "pipeline": 1}


@pytest.fixture
def summary(tmp_path, monkeypatch):
    csrc = tmp_path / "artea_b200" / "csrc"
    csrc.mkdir(parents=True)
    (csrc / "search.cuh").write_text("kernels")
    (tmp_path / "profiles").mkdir()
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))

    def write(source, tuning=TUNING):
        lines = [f"captured_tuning: {json.dumps(tuning)}", "traffic_bytes_per_launch: 1234 (one capture)"]
        if source:
            lines.append(f"captured_source: {source}")
        (tmp_path / "profiles" / "search_kernel_w.md").write_text("\n".join(lines))
    return write


def test_same_kernels(summary):
    summary(bench.search_source())
    assert bench.profile_traffic("w", TUNING, 1.0)[0] == 1234.0


@pytest.mark.parametrize("source", [None, "000000000000"])
def test_other_kernels(summary, source):
    summary(source)
    assert bench.profile_traffic("w", TUNING, 1.0)[0] is None


def test_other_launch(summary):
    summary(bench.search_source(), {"warps_per_cta": 2})
    assert bench.profile_traffic("w", TUNING, 1.0)[0] is None
