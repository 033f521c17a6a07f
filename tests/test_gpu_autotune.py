"""The tangent autotuner's times are those of the kernels, in a process that has not loaded them yet."""
import json
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import json
import numpy as np
from tubularflowiga_b200 import api, meshgen
mesh = api.Mesh(meshgen.straight_tube(1.5e-3, 9e-3, 4, 1, 12).mesh)
for _ in range(2):
    ns = api.NavierStokes(mesh, density=1060.0, viscosity=3.5e-3, dt=2e-3, preconditioner=api.AMG, gmres_restart=4,
                          precision=api.MIXED_BF16X3)
    ns.set_state(np.zeros(4 * mesh.nodes))
    ns.assemble(values=False, rhs=False)
    print(json.dumps(ns.tangent_kernel()))
"""


def test_first_times_do_not_hold_the_kernels_loading():
    """A tangent of this mesh takes about 0.1 ms; loading a kernel between the events added 0.8."""
    out = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    first, second = (json.loads(line) for line in out.stdout.strip().splitlines())
    for name in ("fused_ms", "element_ms", "coefficients_ms"):
        assert 0.0 < first[name] < 3.0 * second[name], (first, second)
