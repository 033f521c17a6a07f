"""Solves in one cooperative launch: the forms that a solve takes by its length, its matrix and its segments.

A solve cut into several launches continues at a restart from what the one launch has there (the iterate and the
tolerances), so it gives the same numbers, bit for bit.  Against separate launches (forced by a wait limit of zero) both
ways stop at 1e-12 of the right-hand side, and solutions agree to 1e-7 (condition numbers up to 1e5, as in the comparison
of the two ways elsewhere); the launch counts say which way ran.
"""
import numpy as np
import pytest

from tests.test_gpu_resident_limits import SETTINGS, rel, solve, system

pytestmark = pytest.mark.gpu

RHO, MU, DT = 1060.0, 3.5e-3, 1e-3


@pytest.fixture(scope="module")
def api():
    from tubularflowiga_b200 import api as a
    return a


@pytest.mark.parametrize("per_launch", [1, 16, 50])
@pytest.mark.parametrize("kind", SETTINGS)
def test_continued_solve_is_the_uncut_one(kind, per_launch):
    ns, _ = system(kind, restart=7)
    solve(ns)                                # (the first one also sets up the preconditioner)
    whole, iterations, once = solve(ns)
    assert iterations > 60 and once <= 2
    ns.set_solve_limits(iterations_per_launch=per_launch)
    update, again, launches = solve(ns)
    assert again == iterations
    cycles = -(-per_launch // 7)             # of a launch: it ends with the cycle that reaches its limit
    assert launches - once == -(-iterations // (7 * cycles)) - 1
    assert np.array_equal(update, whole)


def batch_system(api, restart, precision):
    """Three tubes of uneven length with their segments, and an assembled system."""
    from tubularflowiga_b200 import meshgen
    batch = meshgen.combine_tubes([meshgen.straight_tube(1.5e-3, 9e-3, 4, 1, 12),
                                   meshgen.helical_tube(1e-3, 14e-3, 20e-3, 4, 1, 17),
                                   meshgen.straight_tube(2e-3, 6e-3, 3, 1, 5)], [0.2, 0.15, 0.1])
    ns = api.NavierStokes(api.Mesh(batch.mesh), density=RHO, viscosity=MU, dt=DT, preconditioner=api.AMG,
                          amg_coarse_nodes=60, gmres_restart=restart, precision=precision)
    vmask, pmask, vel = api.batch_boundary_conditions(batch)
    ns.set_dirichlet(vmask, pmask, vel)
    ns.set_tractions({2: 0.0})
    ns.set_segments(batch.node_offset)
    start = api.initial_state(vmask, 0.9 * vel)
    ns.set_state(start, start)
    ns.assemble(values=False, rhs=False)
    ns.apply_dirichlet(values=False, rhs=False)
    return ns


@pytest.mark.parametrize("precision", ["FP64", "FP32_JACOBIAN"])
def test_segments_over_restarts_and_launches(api, precision):
    """Tubes that need several restart cycles and stop in different ones."""
    ns = batch_system(api, 9, getattr(api, precision))
    solve(ns)
    whole, iterations, once = solve(ns)
    assert iterations > 3 * 9 and once == 1
    ns.set_solve_limits(iterations_per_launch=20)
    update, again, launches = solve(ns)
    assert again == iterations and launches > 1
    assert np.array_equal(update, whole)
    ns.set_solve_limits(wait_ns=0)
    update, _, launches = solve(ns)
    assert launches > iterations
    assert rel(update, whole) < 1e-7


@pytest.mark.parametrize("precision, layers", [("FP64", 40), ("FP32_JACOBIAN", 80)])
@pytest.mark.parametrize("preconditioner", ["AMG", "BLOCK_JACOBI"])
def test_matrix_past_the_l2(api, precision, layers, preconditioner):
    """More than 96 MiB of matrix: loaded to leave the L2 first."""
    from perf import cases
    if preconditioner == "BLOCK_JACOBI" and precision != "FP64":
        pytest.skip("the reduced Jacobian needs the AMG")
    tube = cases.long_tube(8, 2, layers, 4 * cases.LAYER)
    mesh = api.Mesh(tube.mesh)
    assert mesh.blocks * 16 * (8 if precision == "FP64" else 4) > 96 << 20
    ns = api.NavierStokes(mesh, density=RHO, viscosity=MU, dt=DT, preconditioner=getattr(api, preconditioner),
                          gmres_restart=30, precision=getattr(api, precision))
    vmask, pmask, vel = api.tube_boundary_conditions(tube, 0.2)
    ns.set_dirichlet(vmask, pmask, vel)
    ns.set_tractions({2: 0.0})
    start = api.initial_state(vmask, 0.9 * vel)
    ns.set_state(start, start)
    ns.assemble(values=False, rhs=False)
    ns.apply_dirichlet(values=False, rhs=False)
    solve(ns)
    whole, iterations, once = solve(ns)
    assert once <= 2
    ns.set_solve_limits(wait_ns=0)
    update, _, launches = solve(ns)
    assert launches > iterations
    assert rel(update, whole) < 1e-7


def test_outlets_in_one_launch(api):
    """The outlets' low-rank term."""
    from tubularflowiga_b200 import meshgen
    y = meshgen.y_bifurcation(parent_layers=5, daughter_layers=4, ax=2, ay=4, ring=1, parent_length=6e-3,
                              daughter_length=5e-3)
    mesh = api.Mesh(y.mesh)
    states, launches = [], []
    for wait in (4_000_000_000, 0):
        ns = api.NavierStokes(mesh, density=RHO, viscosity=MU, dt=DT, preconditioner=api.AMG, gmres_restart=64,
                              precision=api.MIXED_BF16X3, nonlinear_rtol=1e-11, nonlinear_atol=1e-300, max_newton=20,
                              newton_forcing=1)
        ns.set_solve_limits(wait_ns=wait)
        vmask, pmask, vel = api.tube_boundary_conditions(y, 0.2)
        ns.set_dirichlet(vmask, pmask, vel)
        start = api.initial_state(vmask, 0.9 * vel)
        ns.set_state(start, start)
        ns.step_outlets_coupled([api.Outlet.rcr(label, 1e8, 1e-10, 1e9) for label in (2, 3)])
        states.append(ns.get_state())
        launches.append(ns.launches())
    assert 2 * launches[0] < launches[1]
    assert rel(states[1], states[0]) < 1e-7


@pytest.mark.parametrize("fp32", [False, True])
def test_transport_in_one_launch(api, fp32):
    from tubularflowiga_b200 import meshgen
    tube = meshgen.straight_tube(1.5e-3, 0.75e-3 * 11, 3, 2, 11)
    mesh = api.Mesh(tube.mesh)
    params = api.transport_params(diffusion=1e-9, vplus=1.0, kplus=1.0, kminus=0.1, detach_plus=0.5, dt=2e-3, n0_bc=1.0,
                                  nplus_bc=0.5, artificial_diffusion=1e-6, restart=50, gmres_rtol=1e-12,
                                  precision=api.MIXED if fp32 else api.FP64)
    velocity = 0.3 * tube.profile
    launches, iterations = [], []
    for profiling in (False, True):
        solver = api.Transport(mesh, params, velocity, *api.resolve_transport_boundaries(tube.labels, velocity, params))
        solver.set_profiling(profiling)
        before = solver.info()["launches"]
        iterations.append(solver.step(3)["total_iterations"])
        launches.append(solver.info()["launches"] - before)
    # a step: the product with P, the inlet values, the solve; the block inverse on the first; two for the last norm
    assert launches[0] == 3 * 3 + 1 + 2
    assert launches[1] > iterations[1]
