"""Assembly of elements of every basis size, against the oracle: one mesh per size with its own remainders.

The FP64 and the split-BF16 tangent skip what lies past an element's own functions in steps of 4, 8 and 32, so the
sizes lie on both sides of those steps.  Tolerances are those of the parity tests: FP64 1e-12 per field pair (a
thousand-term sum of 1e-16 relative terms), split BF16 1e-4.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

RHO, MU, DT = 1060.0, 3.5e-3, 1e-3


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def thinned(mesh, sizes, seed):
    """`mesh` with the elements cut down to the given numbers of functions (the last ones of each dropped)."""
    from tubularflowiga_b200.ntiga import FlatMesh
    rng = np.random.default_rng(seed)
    conn, rows, cols, vals, offsets = [], [], [], [], [0]
    for e in range(mesh.elements):
        b, t = int(mesh.element_offsets[e]), int(mesh.element_offsets[e + 1])
        keep = np.sort(rng.permutation(t - b)[:min(t - b, sizes[e % len(sizes)])]) + b
        conn.append(mesh.connectivity[keep])
        for a in keep:
            lo, hi = int(mesh.extraction_offsets[a]), int(mesh.extraction_offsets[a + 1])
            rows.append(hi - lo)
            cols.append(mesh.extraction_columns[lo:hi])
            vals.append(mesh.extraction_values[lo:hi])
        offsets.append(offsets[-1] + len(keep))
    used = np.unique(np.concatenate(conn))     # every node needs an element
    number = -np.ones(mesh.nodes, np.int64)
    number[used] = np.arange(len(used))
    return FlatMesh(nodes=len(used), element_offsets=np.array(offsets, np.int32),
                    connectivity=number[np.concatenate(conn)].astype(np.int32),
                    extraction_offsets=np.concatenate([[0], np.cumsum(rows)]).astype(np.int32),
                    extraction_columns=np.concatenate(cols), extraction_values=np.concatenate(vals),
                    bezier_points=mesh.bezier_points.copy(),
                    boundary_labels=-np.ones(6 * mesh.elements, np.int32)).contiguous()


@pytest.mark.parametrize("sizes", [(1, 2, 3), (4, 5, 7, 8), (9, 16, 17), (18, 24, 27), (31, 32, 33), (35, 36, 40, 41),
                                   (48, 49, 63, 64)])
@pytest.mark.parametrize("dt", [0.0, DT])
def test_element_sizes(sizes, dt):
    from tubularflowiga_b200 import api, meshgen
    flat = thinned(meshgen.straight_tube(1.5e-3, 4e-3, 5, 3, 6).mesh, sizes, len(sizes))
    rng = np.random.default_rng(3)
    state, before = (rng.normal(size=(flat.nodes, 4)) * [0.2, 0.2, 0.2, 20.0] for _ in range(2))
    pattern = O.Pattern(flat.nodes, flat.element_offsets, flat.connectivity)
    values, rhs = O.assemble(flat, pattern, state.ravel(), before.ravel(), RHO, MU, dt)
    expected = values.reshape(-1, 4, 4)
    for precision, tolerance in ((api.FP64, 1e-12), (api.MIXED_BF16X3, 1e-4)):
        ns = api.NavierStokes(api.Mesh(flat), density=RHO, viscosity=MU, dt=dt, precision=precision,
                              preconditioner=api.BLOCK_JACOBI if precision == api.FP64 else api.AMG)
        ns.set_state(state.ravel(), before.ravel())
        got, r = ns.assemble()
        got = got.reshape(-1, 4, 4)
        for f in range(4):
            assert rel(r[f::4], rhs[f::4]) < 1e-12
        for i in range(4):
            for f in range(4):
                assert rel(got[:, i, f], expected[:, i, f]) < tolerance, (precision, i, f)
