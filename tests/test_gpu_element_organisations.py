"""Elements of every basis size through every organisation of the tensor-core tangent, against the oracle.

The kernels skip what lies past an element's own functions in steps of 16 (the product) and from 32 down (half of the
warps); a persistent CTA meets items of different sizes one after the other.  Tolerances per field pair are those of the
parity tests: plain BF16 operands 2e-2, split BF16 1e-4, TF32 5e-3.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_gpu_element_sizes import DT, MU, RHO, rel, thinned

pytestmark = pytest.mark.gpu

TOLERANCES = {"MIXED": 2e-2, "MIXED_BF16X3": 1e-4, "MIXED_TF32": 5e-3}


@pytest.fixture(scope="module", params=[(1, 2, 3), (4, 8, 15), (16, 17, 31), (32, 33, 47), (48, 49, 63, 64),
                                        (1, 64, 16, 33, 5, 48)])
def problem(request):
    from tubularflowiga_b200 import api, meshgen
    flat = thinned(meshgen.straight_tube(1.5e-3, 4e-3, 5, 3, 6).mesh, request.param, len(request.param))
    assert 4 * flat.elements > 2 * 2 * 148           # a persistent CTA takes several items
    rng = np.random.default_rng(11)
    state, before = (rng.normal(size=(flat.nodes, 4)) * [0.2, 0.2, 0.2, 20.0] for _ in range(2))
    pattern = O.Pattern(flat.nodes, flat.element_offsets, flat.connectivity)
    values, rhs = O.assemble(flat, pattern, state.ravel(), before.ravel(), RHO, MU, DT)
    return api.Mesh(flat), state.ravel(), before.ravel(), values.reshape(-1, 4, 4), rhs


@pytest.mark.parametrize("precision", TOLERANCES)
@pytest.mark.parametrize("kernel", ["TANGENT_COEFFICIENTS", "TANGENT_FUSED", "TANGENT_ELEMENT"])
def test_sizes_of_every_organisation(problem, kernel, precision):
    from tubularflowiga_b200 import api
    mesh, state, before, expected, rhs = problem
    ns = api.NavierStokes(mesh, density=RHO, viscosity=MU, dt=DT, precision=getattr(api, precision),
                          preconditioner=api.AMG, tangent_kernel=getattr(api, kernel))
    ns.set_state(state, before)
    for _ in range(2):                               # the second assembly reuses what the first left in the chip
        got, r = ns.assemble()
        got = got.reshape(-1, 4, 4)
        for f in range(4):
            assert rel(r[f::4], rhs[f::4]) < 1e-12
        for i in range(4):
            for f in range(4):
                assert rel(got[:, i, f], expected[:, i, f]) < TOLERANCES[precision], (i, f)
