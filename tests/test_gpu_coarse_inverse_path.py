"""Which way the AMG's dense coarse inverse took.

The blocked elimination takes two launches per 32 columns; where it fails, the column-by-column elimination that replaces
it takes two per column, and gives the same inverse.  The launches of a solve that sets the preconditioner up, less those
of the same solve without the set-up, say which one ran, from one partial panel to a cluster of twelve CTAs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core, ring, layers, ctas", [(1, 1, 2, 1), (3, 1, 3, 1), (3, 1, 4, 2), (4, 1, 16, 6),
                                                      (5, 1, 18, 9), (4, 2, 24, 12)])
def test_blocked_inverse_ran(core, ring, layers, ctas):
    from tubularflowiga_b200 import api, meshgen
    tube = meshgen.straight_tube(1.5e-3, 0.5e-3 * layers, core, ring, layers)
    n = 4 * tube.mesh.nodes
    assert (n + 511) // 512 == ctas
    ns = api.NavierStokes(api.Mesh(tube.mesh), density=1060.0, viscosity=3.5e-3, dt=1e-3, preconditioner=api.AMG,
                          amg_coarse_nodes=2048, gmres_restart=20)
    vmask, pmask, vel = api.tube_boundary_conditions(tube, 0.2)
    ns.set_dirichlet(vmask, pmask, vel)
    ns.set_tractions({2: 0.0})
    start = api.initial_state(vmask, vel)
    ns.set_state(start, start)
    ns.assemble(values=False, rhs=False)
    ns.apply_dirichlet(values=False, rhs=False)
    launches, updates = [], []
    for _ in range(2):
        before = ns.launches()
        updates.append(ns.solve_linear(rtol=1e-10, max_iterations=20)[0])
        launches.append(ns.launches() - before)
    assert np.array_equal(updates[0], updates[1])
    # the scattering, the unit order, the panels, the columns' order; Galerkin, A P, unit diagonal, block inverses
    assert launches[0] - launches[1] == 2 * ((n + 31) // 32) + 3 + 4
