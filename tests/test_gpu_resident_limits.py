"""Solves in one cooperative launch at their limits: a barrier wait that runs out.

A wait limit of zero lets every wait run out: the launch ends with its error status, and the solve is done by separate
launches from its start.  Both ways stop at 1e-12 of the right-hand side; as for the same comparison with profiled
(separate) solves, their solutions agree to 1e-7.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SETTINGS = {"block-jacobi": {}, "amg": dict(preconditioner=1, amg_coarse_nodes=40),
            "fp32-jacobian": dict(preconditioner=1, amg_coarse_nodes=40, precision=2),
            "fp32-jacobian-fp64-basis": dict(preconditioner=1, amg_coarse_nodes=40, precision=2, krylov_fp64_basis=1)}


def system(kind, restart=64, layers=9, **settings):
    """A Navier-Stokes handle that holds an assembled linear system, and its tube."""
    from tubularflowiga_b200 import api, meshgen
    assert (api.AMG, api.FP32_JACOBIAN) == (1, 2)
    tube = meshgen.straight_tube(1.5e-3, 0.75e-3 * layers, 3, 1, layers)
    ns = api.NavierStokes(api.Mesh(tube.mesh), density=1060.0, viscosity=3.5e-3, dt=1e-3, gmres_restart=restart,
                          **SETTINGS[kind], **settings)
    vmask, pmask, vel = api.tube_boundary_conditions(tube, 0.2)
    ns.set_dirichlet(vmask, pmask, vel)
    ns.set_tractions({2: 0.0})
    start = api.initial_state(vmask, 0.9 * vel)
    ns.set_state(start, start)
    ns.assemble(values=False, rhs=False)
    ns.apply_dirichlet(values=False, rhs=False)
    return ns, tube


def solve(ns, rtol=1e-12, max_iterations=3000):
    before = ns.launches()
    update, iterations, residual = ns.solve_linear(rtol=rtol, max_iterations=max_iterations)
    return update, iterations, ns.launches() - before


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("kind", SETTINGS)
def test_expired_wait_solves_by_separate_launches(kind):
    ns, _ = system(kind)
    whole, iterations, once = solve(ns)
    assert iterations > 20 and once < iterations
    ns.set_solve_limits(wait_ns=0)
    for _ in range(2):                       # the solve whose wait runs out, and the next one
        update, iterations, launches = solve(ns)
        assert launches > iterations
        assert rel(update, whole) < 1e-7
    ns.set_solve_limits()
    update, iterations, launches = solve(ns)
    assert launches < iterations and rel(update, whole) < 1e-7


def test_expired_wait_of_segments():
    from tubularflowiga_b200 import api, meshgen
    batch = meshgen.combine_tubes([meshgen.straight_tube(1.5e-3, 9e-3, 4, 1, 12),
                                   meshgen.straight_tube(2e-3, 6e-3, 3, 1, 5)], [0.2, 0.1])
    states, launches = [], []
    for wait in (4_000_000_000, 0):
        ns = api.NavierStokes(api.Mesh(batch.mesh), density=1060.0, viscosity=3.5e-3, dt=1e-3, preconditioner=api.AMG,
                              gmres_restart=64, precision=api.MIXED_BF16X3, nonlinear_rtol=1e-11, nonlinear_atol=1e-300,
                              max_newton=20, newton_forcing=1)
        ns.set_solve_limits(wait_ns=wait)
        vmask, pmask, vel = api.batch_boundary_conditions(batch)
        ns.set_dirichlet(vmask, pmask, vel)
        start = api.initial_state(vmask, 0.9 * vel)
        ns.set_state(start, start)
        ns.set_tractions({2: 0.0})
        ns.set_segments(batch.node_offset)
        ns.step()
        states.append(ns.get_state())
        launches.append(ns.launches())
    assert launches[0] < launches[1]
    assert rel(states[1], states[0]) < 1e-7


def test_limits_are_checked():
    from tubularflowiga_b200 import api
    ns, _ = system("block-jacobi")
    for limits in ((0, 1), (-1, 1), (1, -1)):
        with pytest.raises(api.TfigaError):
            ns.set_solve_limits(*limits)
