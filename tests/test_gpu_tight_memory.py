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


HOLE = 32768


class Full:
    """All device memory that cudaMalloc gives, down to pieces of 512 bytes, but for a hole of 32 KiB."""

    def __init__(self):
        import ctypes
        self.runtime = ctypes.CDLL("libcudart.so.12")
        self.runtime.cudaMalloc.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
        self.runtime.cudaFree.argtypes = [ctypes.c_void_p]
        self.pieces = []
        hole, size = self.take(HOLE), 1 << 37
        while size >= 512:
            pointer = self.take(size)
            if pointer is None:
                size //= 2
            else:
                self.pieces.append(pointer)
        self.runtime.cudaFree(hole)

    def take(self, size):
        import ctypes
        pointer = ctypes.c_void_p()
        if self.runtime.cudaMalloc(ctypes.byref(pointer), size) == 0:
            return pointer
        self.runtime.cudaGetLastError()
        return None

    def close(self):
        for p in self.pieces:
            self.runtime.cudaFree(p)


@pytest.mark.parametrize("kind", ["block-jacobi", "amg"])
def test_solve_without_memory_for_its_plan(api, kind):
    """A solve whose one-launch plan finds no memory (the triangular factor alone takes 33 KB) runs as separate launches,
    which need none of the plan's arrays, and holds on to none of them."""
    from tests.test_gpu_resident_limits import solve, system
    ns, _ = system(kind)
    ns.set_profiling(True)                  # separate launches: their arrays and code are there now
    want, iterations, launches = solve(ns)
    ns.set_profiling(False)
    full = Full()
    try:
        update, _, separate = solve(ns)
        hole = full.take(HOLE)
        if hole is not None:
            full.pieces.append(hole)
    finally:
        full.close()
    assert launches > iterations and separate > iterations
    assert rel(update, want) < 1e-7
    assert hole is not None
    ns.set_solve_limits()                   # plans anew
    update, iterations, once = solve(ns)
    assert once < iterations and rel(update, want) < 1e-7
