"""The bench where the reference's CPU functions are neither built nor there as sources:
the reference arm says so in its one line and exits normally, and the GPU arm runs
without its CPU leg instead of losing its measurements to it."""
import importlib.util
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def bench(monkeypatch, tmp_path):
    spec = importlib.util.spec_from_file_location("bench_without_ref", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    monkeypatch.setattr(mod, "REF_LIB", str(tmp_path / "libstref.so"), raising=False)
    from oracle import oracle
    monkeypatch.setattr(oracle, "REF_SRC", str(tmp_path / "src"))
    monkeypatch.setattr(oracle, "HERE", str(tmp_path))
    # a child process would not see these: measured legs must not be reached
    for leg in ("cpu_reference", "cpu_reference_jobs"):
        monkeypatch.setattr(mod, leg, lambda *a, **k: pytest.fail("a CPU leg was started"))
    return mod


def test_reference_arm_says_why(bench, monkeypatch, capsys):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "2", "--warmup", "3"])
    bench.main()
    lines = capsys.readouterr().out.splitlines()
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert set(d) == {"impl", "unavailable"} and d["impl"] == "reference"
    assert d["unavailable"] and "\n" not in d["unavailable"]


def test_gpu_arm_goes_without_the_cpu_leg(bench, monkeypatch):
    seen = []
    monkeypatch.setattr(bench, "run_ours", seen.append)
    monkeypatch.setattr(sys, "argv", ["bench.py"])
    bench.main()
    assert seen[0].no_cpu_baseline and seen[0].cpu_baseline_missing
