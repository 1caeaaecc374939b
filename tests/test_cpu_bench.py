"""bench.py on a host without the reference's driver."""
import argparse
import json
import sys

import pytest


@pytest.fixture
def bench(monkeypatch, tmp_path):
    import bench
    from oracle import run_ref

    monkeypatch.setattr(run_ref, "DRIVER", str(tmp_path / "ref_driver"))
    monkeypatch.setattr(run_ref, "DRIVER_QS", str(tmp_path / "ref_driver_qs"))
    return bench


@pytest.mark.parametrize("workload", ["radix", "bitonic", "join", "batch", "serve", "prims"])
def test_reference_arm_says_why_it_is_unavailable(bench, monkeypatch, capsys, workload):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--workload", workload, "--steps", "1"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "ref_driver" in line["unavailable"] and "value" not in line


@pytest.mark.parametrize("workload", ["radix", "bitonic", "join", "prims"])
def test_own_arm_keeps_its_line_without_a_cpu_baseline(bench, workload):
    """the timed GPU figures are printed whether or not the CPU sample can run"""
    wl = bench.WORKLOADS[workload].__new__(bench.WORKLOADS[workload])
    wl.bits, wl.seed, wl.n, wl.quick = 40, 7, 1024, False
    got = bench.cpu_baseline(wl, argparse.Namespace(cpu_sample=1024))
    assert list(got) == ["unavailable"] and "ref_driver" in got["unavailable"]
