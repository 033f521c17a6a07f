"""The AMG's dense coarse inverse at the edges of its panels, CTAs and clusters.

The coarse space is the mesh itself when it has at most amg_coarse_nodes nodes: the preconditioner is then the exact
inverse (coarse correction) up to rounding, so the flexible GMRES needs one or two iterations and its solution is the
direct one.  Sizes run over one partial panel, one CTA, two CTAs and a cluster that needs the non-portable size.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core, ring, layers", [(1, 1, 2), (2, 1, 3), (3, 1, 4), (3, 1, 7), (4, 1, 16), (4, 2, 24)])
def test_exact_coarse_space_solves_in_one_iteration(core, ring, layers):
    from tubularflowiga_b200 import api, meshgen
    tube = meshgen.straight_tube(1.5e-3, 0.5e-3 * layers, core, ring, layers)
    n = tube.mesh.nodes
    assert n <= 2048
    ns = api.NavierStokes(api.Mesh(tube.mesh), density=1060.0, viscosity=3.5e-3, dt=1e-3, preconditioner=api.AMG,
                          amg_coarse_nodes=2048, gmres_restart=20)
    vmask, pmask, vel = api.tube_boundary_conditions(tube, 0.2)
    ns.set_dirichlet(vmask, pmask, vel)
    ns.set_tractions({2: 0.0})
    start = api.initial_state(vmask, vel)
    ns.set_state(start, start)
    ns.assemble(values=False, rhs=False)
    _, rhs = ns.apply_dirichlet(values=False)
    # the coarse operator drops only the constrained rows and columns, which are identity rows with a zero
    # right-hand side here (the state holds the prescribed values): one application solves the system to the
    # rounding of an inverse of its condition number (about 1e12), 1e-4 of the residual, so 3 iterations reach 1e-10
    update, iterations, residual = ns.solve_linear(rtol=1e-10, max_iterations=20)
    assert iterations <= 4
    assert residual <= 1e-10 * np.linalg.norm(rhs)
    assert np.isfinite(update).all() and np.linalg.norm(update) > 0
