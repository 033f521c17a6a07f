"""Solver handles where little device memory is free (the rest held by this process).

The 12,800-element section's tables take 2.1 GB; a mixed handle's points' numbers 236 MB, or 38 MB a slab.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, MU, DT = 1060.0, 3.5e-3, 2e-3
MB = 1 << 20


@pytest.fixture(scope="module")
def api():
    from tubularflowiga_b200 import api as a
    return a


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def free_bytes():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def hold_all_but(bytes_left):
    """Device memory that this process holds, in one block."""
    import torch
    size = free_bytes() - bytes_left
    assert size > 0
    return torch.empty(size, dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def section(api):
    from perf import cases
    tube = cases.long_tube(8, 2, 100, cases.LAYER)
    return tube, api.Mesh(tube.mesh)


def assemble(api, tube, mesh, **settings):
    """Handle, its device memory after a first assembly, Jacobian and residual."""
    rng = np.random.default_rng(5)
    state = rng.normal(size=(mesh.nodes, 4)) * [0.02, 0.02, 0.02, 5.0]
    state[:, :3] += 0.2 * tube.profile
    before = free_bytes()
    ns = api.NavierStokes(mesh, density=RHO, viscosity=MU, dt=DT, gmres_restart=4, **settings)
    ns.set_state(state.ravel(), state.ravel())
    values, rhs = ns.assemble()
    return ns, before - free_bytes(), values, rhs


@pytest.mark.parametrize("kernel", ["TANGENT_FUSED", "TANGENT_AUTO"])
def test_points_numbers_in_slabs(api, section, kernel):
    """The organisation for meshes that barely fit holds a slab of the points' numbers where memory is short: less than
    11 KiB per element, and the same tangent (FP32 additions in another order) and residual."""
    tube, mesh = section
    elements = tube.mesh.elements
    settings = dict(preconditioner=api.AMG, precision=api.MIXED_BF16X3)
    ns, whole, values, rhs = assemble(api, tube, mesh, tangent_kernel=api.TANGENT_FUSED, **settings)
    del ns
    held = hold_all_but(800 * MB)
    try:
        ns, slabs, got, r = assemble(api, tube, mesh, tangent_kernel=getattr(api, kernel), **settings)
        assert ns.tangent_kernel()["kernel"] == "fused"
        assert whole - slabs > elements * (18 - 11) * 1024
        assert rel(got, values) < 1e-6
        assert rel(r, rhs) < 1e-12
    finally:
        del held
        free_bytes()
