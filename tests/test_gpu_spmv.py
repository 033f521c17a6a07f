"""The 4x4-block product where the split of rows over warps and the loads change.

Rows are shared by four, two or one warps by the number of nodes, and a matrix of more than 96 MB is streamed.  The
products of the device's own Jacobian (downloaded) agree with the same product on the host to 1e-14 of the largest
entry-wise sum of magnitudes: sums of up to 800 products of FP64 numbers in another order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core, ring, layers", [(1, 1, 1), (2, 1, 3), (4, 1, 30), (5, 2, 23), (5, 2, 61), (6, 1, 150)])
@pytest.mark.parametrize("reduced", [False, True])
def test_product_matches_host(core, ring, layers, reduced):
    import torch
    from tubularflowiga_b200 import api, meshgen
    tube = meshgen.straight_tube(1.5e-3, 2e-4 * layers, core, ring, layers)
    mesh = api.Mesh(tube.mesh)
    ns = api.NavierStokes(mesh, density=1060.0, viscosity=3.5e-3, dt=1e-3, gmres_restart=4,
                          preconditioner=api.AMG if reduced else api.BLOCK_JACOBI,
                          precision=api.FP32_JACOBIAN if reduced else api.FP64)
    rng = np.random.default_rng(layers)
    state = rng.normal(size=(mesh.nodes, 4)) * [0.2, 0.2, 0.2, 20.0]
    ns.set_state(state.ravel(), state.ravel())
    values, _ = ns.assemble(rhs=False)
    rows, columns, _ = mesh.pattern()
    x = rng.normal(size=(mesh.nodes, 4))
    blocks = values.reshape(-1, 4, 4)
    def by_rows(b, v):
        products = np.einsum("kij,kj->ki", b, v[columns])
        return np.add.reduceat(products, rows[:-1], axis=0)
    expected, magnitude = by_rows(blocks, x), by_rows(np.abs(blocks), np.abs(x))
    dx = torch.from_numpy(x.ravel().copy()).cuda()
    dy = torch.full((4 * mesh.nodes,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ns.spmv_device(dx.data_ptr(), dy.data_ptr())
    ns.synchronize()
    y = dy.cpu().numpy().reshape(-1, 4)
    assert np.abs(y - expected).max() <= 1e-14 * magnitude.max()
    assert (np.abs(y - expected) <= 1e-12 * magnitude + 1e-300).all()
