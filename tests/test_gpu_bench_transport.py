"""The transport workload of the benchmark, on the 12,800-element section."""
import json
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

STEPS = 2


@pytest.fixture(scope="module")
def line():
    out = subprocess.run([sys.executable, "bench.py", "--workload", "transport", "--transport-mesh", "c2-100", "--steps",
                          str(STEPS), "--warmup", "3", "--no-cpu-baseline", "--no-fp64-leg"], cwd=ROOT,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    return json.loads(out.stdout.strip().splitlines()[-1])


def test_transport_workload_runs(line):
    """The per-family arrays hold every family the library writes (the run once ended in a corrupted heap)."""
    assert line["steps"] == STEPS and line["value"] > 0 and line["e2e"]["value"] > 0
    assert line["kernels"]["spmv_block_jacobi_2x2"]["launches"] > 0


def test_transport_headline_is_not_profiled(line):
    """The headline steps are the ones a caller's program runs: every solve fits one cooperative launch, so a step takes
    a handful of launches (the product with P, the inlet values, the solve) and a profiled one hundreds (about a dozen
    per GMRES iteration).  The kernel figures come from a profiled repeat, and their shares are of that repeat."""
    assert line["gpu_launches"] <= 4 * STEPS
    profiled = line["profile_pass"]
    assert profiled["gpu_launches"] > 10 * line["gpu_launches"]
    assert line["ms_per_step"] < profiled["ms_per_step"]
    assert 0.0 < sum(k["share"] for k in line["kernels"].values()) <= 1.0
