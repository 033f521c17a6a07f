"""The 4x4-block product in every form that the mesh's size selects, and at every remainder of a row's blocks.

Rows are shared by four warps up to 2,368 of them, by two up to 4,736, and have one warp above; a matrix of more than
96 MiB is streamed past the L2, and in FP32 the rows' remainders are taken by twos from 10,065 to 14,208 rows.  The
meshes lie in these ranges (asserted, so that a change of the rule shows), and the rows of a thinned mesh have from 1 to
some 90 blocks.  Products agree with the host's to 1e-14 of the largest entry-wise
sum of magnitudes and 1e-12 of each entry's own (sums of up to 1,372 products of FP64 numbers in another order).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STREAM = 96 << 20
FOUR, TWO = 2368, 4736
PAIRS = range(10065, 14209)


def products(flat, reduced, seed):
    """(device product, host product, product of magnitudes, bytes of the matrix) of a random state's Jacobian."""
    import torch
    from tubularflowiga_b200 import api
    mesh = api.Mesh(flat)
    ns = api.NavierStokes(mesh, density=1060.0, viscosity=3.5e-3, dt=1e-3, gmres_restart=4,
                          preconditioner=api.AMG if reduced else api.BLOCK_JACOBI,
                          precision=api.FP32_JACOBIAN if reduced else api.FP64)
    rng = np.random.default_rng(seed)
    state = rng.normal(size=(mesh.nodes, 4)) * [0.2, 0.2, 0.2, 20.0]
    ns.set_state(state.ravel(), state.ravel())
    values, _ = ns.assemble(rhs=False)
    rows, columns, _ = mesh.pattern()
    x = rng.normal(size=(mesh.nodes, 4))
    blocks = values.reshape(-1, 4, 4)

    def by_rows(b, v):
        return np.add.reduceat(np.einsum("kij,kj->ki", b, v[columns]), rows[:-1], axis=0)

    dx = torch.from_numpy(x.ravel().copy()).cuda()
    dy = torch.full((4 * mesh.nodes,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ns.spmv_device(dx.data_ptr(), dy.data_ptr())
    ns.synchronize()
    return (dy.cpu().numpy().reshape(-1, 4), by_rows(blocks, x), by_rows(np.abs(blocks), np.abs(x)),
            mesh.blocks * 16 * (4 if reduced else 8))


def check(y, expected, magnitude):
    assert np.abs(y - expected).max() <= 1e-14 * magnitude.max()
    assert (np.abs(y - expected) <= 1e-12 * magnitude + 1e-300).all()


@pytest.mark.parametrize("core, ring, layers, reduced, parts, streamed, pairs", [
    (4, 1, 30, False, 4, False, False), (5, 1, 70, False, 2, False, False), (3, 1, 250, False, 1, False, False),
    (6, 1, 100, False, 1, True, False), (6, 1, 140, False, 1, True, False),
    (4, 1, 30, True, 4, False, False), (5, 1, 70, True, 2, False, False), (6, 1, 70, True, 1, False, False),
    (6, 1, 136, True, 1, True, False), (6, 1, 140, True, 1, True, True), (5, 2, 180, True, 1, True, True),
    (8, 2, 100, True, 1, True, False)])
def test_product_of_every_form(core, ring, layers, reduced, parts, streamed, pairs):
    from perf import cases
    flat = cases.long_tube(core, ring, layers, cases.LAYER).mesh
    y, expected, magnitude, size = products(flat, reduced, layers)
    assert parts == (4 if flat.nodes <= FOUR else 2 if flat.nodes <= TWO else 1)
    assert streamed == (size > STREAM)
    assert pairs == (reduced and streamed and flat.nodes in PAIRS)
    check(y, expected, magnitude)


@pytest.mark.parametrize("reduced", [False, True])
def test_product_of_short_rows(reduced):
    from tests.test_gpu_element_sizes import thinned
    from tubularflowiga_b200 import meshgen
    flat = thinned(meshgen.straight_tube(1.5e-3, 4e-3, 5, 3, 12).mesh, tuple(range(1, 14)), 4)
    y, expected, magnitude, _ = products(flat, reduced, 7)
    check(y, expected, magnitude)
