"""bench.py where the reference's own library is not there: both arms print their line all the same."""
import argparse
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture
def bench(monkeypatch):
    import bench as b
    from oracle.oracle import Ref

    def missing():
        raise RuntimeError("the reference harness is not built\n(no reference tree)")

    monkeypatch.setattr(Ref, "lib", staticmethod(missing))
    return b


def test_the_figure_beside_is_null(bench):
    def measure():
        raise AssertionError("not reached")

    assert bench.beside(measure) == {"cpu_baseline": None,
                                     "cpu_baseline_unavailable": "the reference harness is not built (no reference tree)"}


@pytest.mark.parametrize("workload", ["six_sensors", "sink_evt3_1280x720"])
def test_the_reference_arm_says_why(bench, workload):
    out = bench.run_reference(argparse.Namespace(workload=workload, warmup=1, steps=1, gpus=1, cpu_windows=1), 0)
    assert out == {"impl": "reference", "unavailable": "the reference harness is not built (no reference tree)"}
    assert bench.run_reference(argparse.Namespace(workload=workload), 1) is None


def test_the_command_line():
    from oracle.oracle import Ref

    if Ref.available():
        pytest.skip("the reference harness is built here")
    r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference"], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "\n" not in line["unavailable"] and line["unavailable"]
