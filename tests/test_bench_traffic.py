"""The bench's DRAM traffic comes from the committed profile of the kernel that ran, or is not reported."""
import importlib
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def bench(monkeypatch, tmp_path):
    monkeypatch.syspath_prepend(ROOT)
    b = importlib.import_module("bench")
    (tmp_path / "profiles").mkdir()
    (tmp_path / "profiles" / "upwind_sweep_mesh7.md").write_text(
        "text\n| upwind_sweep | k_sweep, mesh7 | traffic_bytes_per_launch=1.5e9 |\n"
        "| upwind_sweep | k_sweep_staged, mesh7 | traffic_bytes_per_launch=2.5e9 |\n"
        "| other | mesh7 | traffic_bytes_per_launch=7 |\n")
    monkeypatch.setattr(b, "ROOT", str(tmp_path))
    return b


def test_traffic_of_the_kernel_that_ran(bench):
    assert bench.ncu_traffic("upwind_sweep", "mesh7", "k_sweep")[0] == 1.5e9
    assert bench.ncu_traffic("upwind_sweep", "mesh7", "k_sweep_staged")[0] == 2.5e9
    assert bench.ncu_traffic("upwind_sweep", "mesh7", "k_sweep_stream") == (None, None)
    assert bench.ncu_traffic("other", "mesh7")[0] == 7
    assert bench.ncu_traffic("other", "mesh8") == (None, None)


def test_committed_profiles_name_the_sweep_kernel():
    sys.path.insert(0, ROOT)
    try:
        b = importlib.import_module("bench")
    finally:
        sys.path.remove(ROOT)
    for workload in ("square100k", "square20k"):
        value, path = b.ncu_traffic("upwind_sweep", workload, "k_sweep_stream")
        assert value and path
