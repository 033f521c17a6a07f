"""What users of this framework have it compute, as cases that can be timed and compared.

A case is one pass through the public binding (``tubularflowiga_b200.api``) on a generated mesh:

* ``spmv``       the 4x4-block product with an assembled Jacobian on device vectors;
* ``tangent``    residual and exact Newton tangent of a given state;
* ``solve``      one linear system of a Newton iteration, by the default block-Jacobi GMRES;
* ``step``       a backward-Euler step to convergence: one tube, a Y-bifurcation with RCR outlets, a batch;
* ``transport``  a two-species transport run: matrices, time steps, final state.

Meshes are O-grid tubes of ``core``^2 + 4 ``core`` ``ring`` elements a layer, as the benchmark's, or small
relatives of its Y-bifurcation and its batch of tubes.  Fluid, time steps and solver settings are the benchmark's;
``precision`` is the plain FP64 solver or the split-BF16 mixed one that the benchmark runs by default.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tubularflowiga_b200 import api, meshgen
from tubularflowiga_b200.ntiga import FlatMesh

RHO, MU = 1060.0, 3.5e-3                       # blood, SI units
RADIUS = 1.5e-3
TRANSPORT = dict(diffusion=1e-9, vplus=1.0, kplus=1.0, kminus=0.1, detach_plus=0.5, dt=2e-3, n0_bc=1.0, nplus_bc=0.5,
                 artificial_diffusion=1e-6)
RCR = (1e8, 1e-10, 1e9)                        # proximal resistance, capacitance, distal resistance
LAYER = RADIUS / 20                            # axial element length of the 51,200-element pulsatile tube
PRECISION = {"fp64": 0, "fp32-jacobian": 2, "bf16x3": 3}


def listed():
    """The cylinder (1,280 elements) is the smallest configuration, where launches and latency count; the 12,800
    element section of the pulsatile tube is an ordinary one; 25,600 elements fill the chip many times over."""
    cylinder = dict(geometry="tube", core=4, ring=1, layers=40, layer_length=10 * LAYER)
    section = dict(geometry="tube", core=8, ring=2, layers=100, layer_length=LAYER)
    return [
        # what a program that brings its own Krylov method calls in its inner loop: small, and streaming from HBM
        dict(name="spmv cylinder fp64", kind="spmv", precision="fp64", dt=1e-3, **cylinder),
        dict(name="spmv section fp32", kind="spmv", precision="fp32-jacobian", dt=2e-3, **section),
        # one assembly: a steady solve of the cylinder, the plain FP64 solver, and the mixed solver's tangent on a
        # ragged branching mesh and on the largest tube
        dict(name="tangent cylinder fp64", kind="tangent", precision="fp64", dt=0.0, **cylinder),
        dict(name="tangent section fp64", kind="tangent", precision="fp64", dt=2e-3, **section),
        dict(name="tangent bifurcation bf16x3", kind="tangent", precision="bf16x3", dt=2e-3, geometry="bifurcation",
             core=2, ring=2, layers=27, layer_length=4 * LAYER),
        dict(name="tangent long tube bf16x3", kind="tangent", precision="bf16x3", dt=2e-3,
             **dict(section, layers=200)),
        # the reference's own linear solver, this framework's default
        dict(name="solve cylinder fp64", kind="solve", precision="fp64", dt=1e-3, **cylinder),
        # time steps: the FP64 solver on the smallest mesh, then the mixed solver as the benchmark runs it, on one
        # tube, with outlets coupled inside Newton, and on a batch of independent tubes
        dict(name="step cylinder fp64", kind="step", precision="fp64", dt=1e-3, **cylinder),
        dict(name="step section bf16x3", kind="step", precision="bf16x3", dt=2e-3, **section),
        dict(name="step bifurcation bf16x3", kind="step", precision="bf16x3", dt=2e-3, geometry="bifurcation",
             core=2, ring=2, layers=27, layer_length=4 * LAYER),
        dict(name="step batch bf16x3", kind="step", precision="bf16x3", dt=1e-4, geometry="batch", core=4, ring=1,
             layers=60, tubes=5),
        # a transport run on a flow that is known, from its matrices to its last state
        dict(name="transport section fp32", kind="transport", precision="bf16x3", steps=4, **section),
    ]


def draw(rng):
    """A case of the same kinds; cross-sections of 9 to 128 elements a layer, odd ones among them."""
    kind = rng.choice(["spmv", "spmv", "tangent", "tangent", "tangent", "solve", "step", "step", "transport"])
    core, ring = rng.choice([(3, 1), (4, 1), (5, 1), (5, 2), (6, 1), (7, 2), (8, 2)])
    per_layer = core * core + 4 * core * ring
    most = {"spmv": 12800, "tangent": 25600, "solve": 1600, "step": 8000, "transport": 10000}[kind]
    elements = math.exp(rng.uniform(math.log(700), math.log(most)))
    precision = rng.choice(["fp64", "bf16x3"])
    if kind == "tangent" and precision == "fp64":
        elements = min(elements, 12800)
    case = dict(kind=kind, geometry="tube", core=core, ring=ring,
                layers=max(8, min(most // per_layer, round(elements / per_layer))),
                layer_length=LAYER * rng.uniform(1.0, 4.0), dt=rng.choice([1e-3, 2e-3]), precision=precision)
    if kind == "spmv" and case["precision"] == "bf16x3":
        case["precision"] = "fp32-jacobian"
    if kind == "solve":
        case["precision"] = "fp64"             # the mixed solver refuses block-Jacobi
    if kind == "tangent" and rng.random() < 0.3:
        case["dt"] = 0.0
    if kind == "step" and rng.random() < 0.5:
        case["geometry"] = rng.choice(["bifurcation", "batch"])
        if case["geometry"] == "batch":
            case.update(core=4, ring=1, layers=rng.randint(20, 70), tubes=rng.randint(2, 6), dt=1e-4)
        else:
            case.update(core=rng.choice([2, 3]), ring=rng.choice([1, 2]), layers=rng.randint(12, 27))
    if kind == "transport":
        case["steps"] = rng.randint(1, 5)
        del case["dt"]
    return case


# Meshes ----------------------------------------------------------------------------------------------------------


def long_tube(core, ring, layers, layer_length):
    """meshgen.straight_tube with the interior layers, which are translates of one another, copied."""
    base = meshgen.straight_tube(RADIUS, 7 * layer_length, core, ring, 7)
    m, plane, cells = base.mesh, base.per_plane, base.mesh.elements // 7
    shift = np.concatenate([np.zeros(4), np.arange(1, layers - 6), np.full(3, layers - 7)]).astype(np.int64)
    source = np.concatenate([np.arange(4), np.full(layers - 7, 3), np.arange(4, 7)]).astype(np.int64)
    element = lambda k: slice(k * cells, (k + 1) * cells)                              # noqa: E731
    basis = lambda k: slice(m.element_offsets[k * cells], m.element_offsets[(k + 1) * cells])   # noqa: E731
    entry = lambda k: slice(m.extraction_offsets[basis(k).start], m.extraction_offsets[basis(k).stop])  # noqa: E731
    conn, rows, columns, values, points, labels, nen = [], [], [], [], [], [], []
    bezier = m.bezier_points.reshape(-1, 64, 3)
    lengths, sizes = np.diff(m.extraction_offsets), np.diff(m.element_offsets)
    for k, s in zip(source, shift):
        conn.append(m.connectivity[basis(k)] + s * plane)
        rows.append(lengths[basis(k)])
        columns.append(m.extraction_columns[entry(k)])
        values.append(m.extraction_values[entry(k)])
        points.append(bezier[element(k)] + np.array([0.0, 0.0, s * layer_length]))
        labels.append(m.boundary_labels.reshape(-1, 6)[element(k)])
        nen.append(sizes[element(k)])
    offsets = lambda parts: np.concatenate([[0], np.cumsum(np.concatenate(parts))]).astype(np.int32)  # noqa: E731
    mesh = FlatMesh(nodes=plane * (layers + 1), element_offsets=offsets(nen), connectivity=np.concatenate(conn),
                    extraction_offsets=offsets(rows), extraction_columns=np.concatenate(columns),
                    extraction_values=np.concatenate(values), bezier_points=np.concatenate(points).ravel(),
                    boundary_labels=np.concatenate(labels).ravel()).contiguous()
    middle = (slice(plane, 2 * plane), layers - 7)
    stretch = lambda a: np.concatenate([a[:plane * 4], np.tile(a[middle[0]], (middle[1],) + (1,) * (a.ndim - 1)),  # noqa: E731
                                        a[plane * 4:]])
    z = np.repeat(np.arange(layers + 1) * layer_length, plane)
    control = np.concatenate([stretch(base.points)[:, :2], z[:, None]], axis=1)
    return meshgen.Tube(mesh=mesh, points=control, labels=stretch(base.labels), cells=None,
                        profile=stretch(base.profile), radius=RADIUS, length=layers * layer_length,
                        planes=layers + 1, per_plane=plane)


@functools.lru_cache(maxsize=3)
def mesh_of(geometry, core, ring, layers, layer_length, tubes):
    if geometry == "tube":
        return long_tube(core, ring, layers, layer_length)
    if geometry == "bifurcation":
        return meshgen.y_bifurcation(ax=core, ay=2 * core, ring=ring, parent_layers=layers, daughter_layers=layers - 3,
                                     parent_length=layers * layer_length, daughter_length=(layers - 3) * layer_length)
    sizes = np.linspace(0.3, 1.0, tubes)
    parts = []
    for k, size in enumerate(sizes):           # straight and helical tubes of uneven sizes
        radius, n = RADIUS * (0.6 + 0.2 * k), max(8, int(layers * size))
        parts.append(meshgen.straight_tube(radius, 14 * radius, core, ring, n) if k % 2 == 0 else
                     meshgen.helical_tube(radius, 14 * radius, 20e-3, core, ring, n))
    return meshgen.combine_tubes(parts, [0.25 - 0.03 * k for k in range(tubes)])


def geometry_of(case):
    return mesh_of(case["geometry"], case["core"], case["ring"], case["layers"], case.get("layer_length", 0.0),
                   case.get("tubes", 1))


def inflow(case, body, seed):
    """Velocity mask and the seeded inflow velocities at two times one step apart."""
    rng = np.random.default_rng(seed)
    if case["geometry"] == "batch":
        first = rng.uniform(0.8, 1.2, case["tubes"])
        now = first * rng.uniform(1.0, 1.05, case["tubes"])
        return tuple(api.batch_boundary_conditions(body, f)[k] for f, k in ((first, 0), (first, 2), (now, 2)))
    scale = rng.uniform(0.12, 0.22)
    vmask, _, profile = api.tube_boundary_conditions(body, 1.0)
    return vmask, scale * profile, scale * rng.uniform(1.0, 1.1) * profile


def flow_state(body, seed):
    """A developed profile with a disturbance, its pressure falling along the tube: [n, 4]."""
    rng = np.random.default_rng(seed)
    n = body.mesh.nodes
    state = rng.normal(size=(n, 4)) * [0.02, 0.02, 0.02, 5.0]
    state[:, :3] += 0.2 * body.profile
    state[:, 3] += 40.0 * (1.0 - np.arange(n) / n)
    return state


# A pass ------------------------------------------------------------------------------------------------------------


class DeviceBuffer:
    """A handle's device array of doubles, for torch.as_tensor; the tensor keeps the handle that owns it."""

    def __init__(self, owner, pointer, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (pointer, False), "version": 3}


def prepare(case, seed):
    body = geometry_of(case)
    mesh = api.Mesh(body.mesh)
    return {"spmv": prepare_tangent, "tangent": prepare_tangent, "solve": prepare_solve, "step": prepare_step,
            "transport": prepare_transport}[case["kind"]](case, seed, body, mesh)


def prepare_tangent(case, seed, body, mesh):
    n = mesh.nodes
    reduced = case["precision"] != "fp64"
    ns = api.NavierStokes(mesh, density=RHO, viscosity=MU, dt=case["dt"], precision=PRECISION[case["precision"]],
                          preconditioner=api.AMG if reduced else api.BLOCK_JACOBI, gmres_restart=64)
    ns.set_state(flow_state(body, seed), flow_state(body, seed + 1))
    values, _, rhs = ns.device_buffers()
    state = {"case": case, "ns": ns, "x": torch.from_numpy(flow_state(body, seed + 2).ravel()).cuda(),
             "y": torch.empty(4 * n, dtype=torch.float64, device="cuda"),
             "rhs": torch.as_tensor(DeviceBuffer(ns, rhs, 4 * n), device="cuda"),
             "stream": torch.cuda.ExternalStream(ns.stream())}
    if not reduced:
        state["values"] = torch.as_tensor(DeviceBuffer(ns, values, 16 * mesh.blocks), device="cuda")
    if case["kind"] == "spmv":
        ns.assemble(values=False, rhs=False)
    return state


def prepare_solve(case, seed, body, mesh):
    ns = api.NavierStokes(mesh, density=RHO, viscosity=MU, dt=case["dt"])
    vmask, first, inlet = inflow(case, body, seed)
    ns.set_dirichlet(vmask, None, inlet)
    ns.set_tractions({2: 0.0})
    start = api.initial_state(vmask, first)
    ns.set_state(start, start)
    ns.assemble(values=False, rhs=False)
    ns.apply_dirichlet(values=False, rhs=False)
    return {"case": case, "ns": ns}


def prepare_step(case, seed, body, mesh):
    settings = dict(density=RHO, viscosity=MU, dt=case["dt"], precision=PRECISION[case["precision"]],
                    preconditioner=api.AMG, nonlinear_rtol=1e-11, nonlinear_atol=1e-300, max_newton=20,
                    gmres_rtol=1e-12 if case["precision"] == "fp64" else 1e-8, gmres_restart=64)
    if case["precision"] != "fp64":
        settings.update(newton_forcing=1, tangent_reuse_factor=100.0, amg_coarse_period=3)
    ns = api.NavierStokes(mesh, **settings)
    vmask, first, inlet = inflow(case, body, seed)
    ns.set_dirichlet(vmask, None, inlet)
    if case["geometry"] != "bifurcation":
        ns.set_tractions({2: 0.0})
    if case["geometry"] == "batch":
        ns.set_segments(body.node_offset)
    return {"case": case, "ns": ns, "start": api.initial_state(vmask, first), "inlet": inlet.ravel()}


def poiseuille(case, body, seed):
    return np.random.default_rng(seed).uniform(0.2, 0.4) * body.profile


def prepare_transport(case, seed, body, mesh):
    velocity = poiseuille(case, body, seed)
    params = api.transport_params(steps=case["steps"], restart=50, gmres_rtol=1e-11,
                                  precision=api.MIXED if case["precision"] == "bf16x3" else api.FP64, **TRANSPORT)
    return {"case": case, "mesh": mesh, "params": params, "velocity": velocity,
            "boundaries": api.resolve_transport_boundaries(body.labels, velocity, params)}


def run(state):
    case = state["case"]
    if case["kind"] == "transport":
        solver = api.Transport(state["mesh"], state["params"], state["velocity"], *state["boundaries"])
        solver.step(case["steps"])
        out = solver.get_state()
        solver.close()
        return {"species": out}
    ns = state["ns"]
    if case["kind"] == "spmv":
        ns.spmv_device(state["x"].data_ptr(), state["y"].data_ptr())
        return {"product": state["y"]}
    if case["kind"] == "tangent":
        ns.assemble(values=False, rhs=False)
        if "values" in state:
            return {"residual": state["rhs"], "jacobian": state["values"]}
        # the mixed Jacobian stays in the handle, in FP32: what a caller sees of it is its product
        ns.spmv_device(state["x"].data_ptr(), state["y"].data_ptr())
        with torch.cuda.stream(state["stream"]):
            return {"residual": state["rhs"], "jacobian_x": state["y"].float()}
    if case["kind"] == "solve":
        return {"update": ns.solve_linear(rtol=1e-13, max_iterations=20000)[0]}
    ns.set_state(state["start"], state["start"])
    ns.set_dirichlet_values(state["inlet"])
    if case["geometry"] == "bifurcation":
        outlets = [api.Outlet.rcr(label, *RCR) for label in (2, 3)]
        ns.step_outlets_coupled(outlets)
    else:
        ns.step()
    out = ns.get_state().reshape(-1, 4)
    return {"velocity": out[:, :3], "pressure": out[:, 3]}


def work(case):
    """Each array of the mesh and the matrix that a pass needs, once; a solve counts as 32 Krylov iterations, a step as
    one Newton iteration with its solve and the residual that ends it, a transport step as 40 iterations."""
    body = geometry_of(case)
    m = body.mesh
    nen = np.diff(m.element_offsets).astype(np.float64)
    n, pairs = m.nodes, float((nen ** 2).sum())
    blocks = float(block_count(case))
    value = 8 if case["precision"] == "fp64" else 4
    product = {"bytes": blocks * (16 * value + 4) + 64 * n, "flops": 32 * blocks}
    if case["kind"] == "spmv":
        return product
    if case["kind"] == "transport":
        assembly = {"bytes": 4 * 64 * 8 * nen.sum() + 2 * 32 * blocks, "flops": 2 * 64 * 6 * pairs}
        sweep = {"bytes": blocks * (4 * value + 4) + 32 * n, "flops": 8 * blocks}
        return {k: assembly[k] + 40 * case["steps"] * sweep[k] for k in assembly}
    tables = 5 * 64 * 8 * nen.sum()
    tangent = {"bytes": tables + 4 * pairs + 16 * value * blocks + 96 * n, "flops": 8192 * pairs}
    if case["kind"] == "tangent":
        return tangent
    krylov = {k: 32 * product[k] for k in product}
    if case["kind"] == "solve":
        return krylov
    return {k: tangent[k] + krylov[k] + (tables if k == "bytes" else 0) for k in tangent}


@functools.lru_cache(maxsize=64)
def block_count_of(geometry, core, ring, layers, layer_length, tubes):
    count = lambda n: sum(len(np.unique(k)) for k in pair_keys(                         # noqa: E731
        mesh_of(geometry, core, ring, n, layer_length, tubes).mesh))
    if geometry != "tube" or layers < 12:
        return count(layers)
    ten, eleven = count(10), count(11)         # every further layer of a tube adds the same blocks
    return ten + (layers - 10) * (eleven - ten)


def block_count(case):
    return block_count_of(case["geometry"], case["core"], case["ring"], case["layers"], case.get("layer_length", 0.0),
                          case.get("tubes", 1))


def pair_keys(m, rows_at_once=2000):
    """Keys row * nodes + column of all pairs, by slices of the rows."""
    offsets, conn = m.element_offsets.astype(np.int64), m.connectivity.astype(np.int64)
    nen = np.diff(offsets)
    element_of = np.repeat(np.arange(m.elements), nen)
    order = np.argsort(conn, kind="stable")
    starts = np.searchsorted(conn[order], np.arange(0, m.nodes + rows_at_once, rows_at_once))
    for lo, hi in zip(starts[:-1], starts[1:]):
        picked = order[lo:hi]
        count = nen[element_of[picked]]
        first = np.repeat(offsets[element_of[picked]], count)
        within = np.arange(count.sum()) - np.repeat(np.cumsum(count) - count, count)
        yield np.repeat(conn[picked], count) * m.nodes + conn[first + within]


# The same results in plain FP64 torch --------------------------------------------------------------------------------


def bernstein(t):
    """Cubic Bernstein values, first and second derivatives at t: three [len(t), 4]."""
    t = torch.as_tensor(t, dtype=torch.float64)[:, None]
    k = torch.tensor([1.0, 3.0, 3.0, 1.0], dtype=torch.float64)
    i = torch.arange(4.0, dtype=torch.float64)
    power = lambda e, d: (torch.where(e >= d, e, d) - d).clamp(min=0)                   # noqa: E731
    fall = lambda e, d: e if d == 1 else e * (e - 1)                                    # noqa: E731
    p = lambda d: t ** power(i, d) * (fall(i, d) if d else 1.0)                         # noqa: E731
    q = lambda d: (1 - t) ** power(3 - i, d) * ((-1) ** d * fall(3 - i, d) if d else 1.0)   # noqa: E731
    return k * p(0) * q(0), k * (p(1) * q(0) + p(0) * q(1)), k * (p(2) * q(0) + 2 * p(1) * q(1) + p(0) * q(2))


def bezier_basis(points):
    """Values [P, 64], parametric gradient [P, 64, 3] and Hessian [P, 64, 3, 3] of the tricubic Bezier functions."""
    one = [bernstein(points[:, d]) for d in range(3)]
    f = lambda *order: torch.einsum("pk,pj,pi->pkji", one[2][order[2]], one[1][order[1]],  # noqa: E731
                                    one[0][order[0]]).reshape(len(points), 64)
    unit = np.eye(3, dtype=int)
    gradient = torch.stack([f(*unit[a]) for a in range(3)], -1)
    hessian = torch.stack([torch.stack([f(*(unit[a] + unit[b])) for b in range(3)], -1) for a in range(3)], -2)
    return f(0, 0, 0), gradient, hessian


GAUSS, WEIGHT = np.polynomial.legendre.leggauss(4)
GAUSS, WEIGHT = (GAUSS + 1) / 2, WEIGHT / 2


class Elements:
    """A slice of a mesh's elements, their 64-wide dense extraction, and the features N, grad N, Lap N at the 4x4x4
    Gauss points: phi [E, 5, 64 points, 64 functions]; unused functions are zero and point at node 0."""

    def __init__(self, m, lo, hi):
        b, t = int(m.element_offsets[lo]), int(m.element_offsets[hi])
        nen = np.diff(m.element_offsets[lo:hi + 1])
        rows = np.concatenate([64 * k + np.arange(c) for k, c in enumerate(nen)])
        dense = np.zeros(((hi - lo) * 64, 64))
        x0, x1 = int(m.extraction_offsets[b]), int(m.extraction_offsets[t])
        dense[np.repeat(rows, np.diff(m.extraction_offsets[b:t + 1])), m.extraction_columns[x0:x1]] = \
            m.extraction_values[x0:x1]
        nodes = np.zeros((hi - lo) * 64, np.int64)
        nodes[rows] = m.connectivity[b:t]
        used = np.zeros((hi - lo) * 64)
        used[rows] = 1.0
        self.used = torch.from_numpy(used.reshape(-1, 64)).cuda()
        self.nodes = torch.from_numpy(nodes.reshape(-1, 64)).cuda()
        extraction = torch.from_numpy(dense.reshape(-1, 64, 64)).cuda()
        points = torch.from_numpy(m.bezier_points.reshape(-1, 64, 3)[lo:hi]).cuda()
        u = np.stack(np.meshgrid(GAUSS, GAUSS, GAUSS, indexing="ij"), -1).reshape(-1, 3)[:, ::-1]
        weight = torch.from_numpy(np.einsum("i,j,k->ijk", WEIGHT, WEIGHT, WEIGHT).ravel()).cuda()
        value, gradient, hessian = (x.cuda() for x in bezier_basis(torch.from_numpy(u.copy())))
        jacobian = torch.einsum("ekx,qka->eqxa", points, gradient)
        second = torch.einsum("ekx,qkab->eqxab", points, hessian)
        inverse = torch.linalg.inv(jacobian)                                  # [a, x]
        metric = inverse @ inverse.transpose(-1, -2)
        lap = torch.einsum("qkab,eqab->eqk", hessian, metric) - torch.einsum(
            "qkc,eqcx,eqxab,eqab->eqk", gradient, inverse, second, metric)
        grad = torch.einsum("qka,eqax->eqxk", gradient, inverse)
        features = torch.cat([value[None, :, None].expand(hi - lo, -1, 1, -1), grad, lap[:, :, None]], 2)
        self.phi = torch.einsum("eqtk,eak->eqta", features, extraction)       # [E, q, 5, a]
        self.weight = weight * torch.linalg.det(jacobian)
        self.G = inverse.transpose(-1, -2) @ inverse
        self.direction = inverse.sum(2).square().sum(-1)

    def at_points(self, state):
        """Features of a nodal state [n, 4]: [E, q, 5, 4]."""
        return torch.einsum("eqta,eaf->eqtf", self.phi, state[self.nodes] * self.used[..., None])


def slices(m, at_once=800):
    for lo in range(0, m.elements, at_once):
        yield Elements(m, lo, min(m.elements, lo + at_once))


def flux(features, before, G, direction, dt):
    """VMS Navier-Stokes at one point: the factor of (N, grad N) in the weak form of each equation, [4, 4]."""
    u, gu, lap = features[0, :3], features[1:4, :3], features[4, :3]          # gu[d, c] = du_c/dx_d
    p, gp = features[0, 3], features[1:4, 3]
    rate = (u - before) / dt if dt > 0 else torch.zeros_like(u)
    nu = MU / RHO
    tau = (4.0 / dt ** 2 if dt > 0 else 0.0) + u @ G @ u + nu ** 2 / 12.0 * (G * G).sum()
    tau = tau.rsqrt()
    fine = -tau * (rate + u @ gu + gp / RHO - nu * lap)
    divergence = gu.diagonal().sum()
    pressure = p - RHO / (tau * direction) * divergence
    moved = u + fine
    momentum = torch.cat([RHO * (rate + moved @ gu)[None],
                          MU * (gu + gu.T) - RHO * torch.outer(moved, fine)
                          - pressure * torch.eye(3, dtype=u.dtype, device=u.device)])
    return torch.cat([momentum, torch.cat([divergence[None], -fine])[:, None]], 1)


def over_points(f, el, features, before, dt):
    g = torch.func.vmap(torch.func.vmap(lambda a, b, c, d: f(a, b, c, d, dt)))
    return g(features, before, el.G, el.direction)


def exact_assembly(m, state, before, dt, wanted, x=None):
    """rhs [4n], and as `wanted` says the product J x, the 4x4 blocks of J by row-major pairs, or J as a matrix."""
    n = m.nodes
    state, before = (torch.as_tensor(s, dtype=torch.float64).cuda().reshape(n, 4) for s in (state, before))
    rhs = torch.zeros(n, 4, dtype=torch.float64, device="cuda")
    out = None
    if wanted == "product":
        out = torch.zeros_like(rhs)
        x = torch.as_tensor(x, dtype=torch.float64).cuda().reshape(n, 4)
    elif wanted == "matrix":
        out = torch.zeros(n, 4, n, 4, dtype=torch.float64, device="cuda")
    elif wanted == "blocks":
        keys = torch.cat([torch.from_numpy(np.unique(k)) for k in pair_keys(m)]).cuda()
        out = torch.zeros(len(keys), 16, dtype=torch.float64, device="cuda")
    for el in slices(m, 800 if wanted in ("product", None) else 200):
        features, old = el.at_points(state), el.at_points(before)[:, :, 0, :3]
        test = el.phi[:, :, :4] * el.weight[:, :, None, None]
        scatter = lambda to, r: to.index_put_((el.nodes,), r * el.used[..., None], accumulate=True)  # noqa: E731
        scatter(rhs, -torch.einsum("eqsa,eqsi->eai", test, over_points(flux, el, features, old, dt)))
        if wanted is None:
            continue
        tangent = over_points(torch.func.jacfwd(flux), el, features, old, dt)  # [E, q, s, i, t, f]
        if wanted == "product":
            change = torch.einsum("eqsitf,eqtf->eqsi", tangent, el.at_points(x))
            scatter(out, torch.einsum("eqsa,eqsi->eai", test, change))
            continue
        trial = torch.einsum("eqsitf,eqtb->eqsibf", tangent, el.phi)
        block = torch.einsum("eqsa,eqsibf->eabif", test, trial)
        block = block * (el.used[:, :, None] * el.used[:, None, :])[..., None, None]
        if wanted == "matrix":
            flat = (el.nodes[:, :, None] * n + el.nodes[:, None, :]).reshape(-1)
            view = out.permute(0, 2, 1, 3)
            view.index_put_((flat // n, flat % n), block.reshape(-1, 4, 4), accumulate=True)
        else:
            pair = (el.used[:, :, None] * el.used[:, None, :]).reshape(-1) > 0
            flat = (el.nodes[:, :, None] * n + el.nodes[:, None, :]).reshape(-1)[pair]
            out.index_add_(0, torch.searchsorted(keys, flat), block.reshape(-1, 16)[pair])
    return rhs.reshape(-1), (out if out is None else out.reshape(-1) if wanted != "matrix" else out.reshape(4 * n, 4 * n))


def constrained(vmask):
    fixed = np.zeros((len(vmask), 4), bool)
    fixed[:, :3] = np.asarray(vmask)[:, None] != 0
    return torch.from_numpy(fixed.ravel()).cuda()


def exact(case, seed):
    body = geometry_of(case)
    m, kind = body.mesh, case["kind"]
    if kind == "transport":
        return exact_transport(case, seed, body) if m.nodes <= 15000 else None
    if kind in ("spmv", "tangent"):
        state, before, x = (flow_state(body, seed + k) for k in range(3))
        if kind == "tangent" and case["precision"] == "fp64":
            rhs, jacobian = exact_assembly(m, state, before, case["dt"], "blocks")
            return {"residual": rhs, "jacobian": jacobian}
        rhs, product = exact_assembly(m, state, before, case["dt"], "product", x)
        return {"residual": rhs, "jacobian_x": product} if kind == "tangent" else {"product": product}
    if case["geometry"] == "bifurcation":      # its outlets' fixed point needs dense solves of the whole mesh
        return None
    vmask, first, inlet = inflow(case, body, seed)
    start = api.initial_state(vmask, first)
    parts = [(m, slice(0, m.nodes))]
    if case["geometry"] == "batch":
        parts = [(t.mesh, slice(a, b)) for t, a, b in zip(body.tubes, body.node_offset[:-1], body.node_offset[1:])]
    if max(p.nodes for p, _ in parts) > 4500:
        return None
    found = [exact_flow(p, vmask[s], inlet[s], start.reshape(-1, 4)[s], case["dt"], kind) for p, s in parts]
    out = torch.cat(found)
    return {"update": out.reshape(-1)} if kind == "solve" else {"velocity": out[:, :3], "pressure": out[:, 3]}


def exact_flow(m, vmask, inlet, start, dt, kind):
    """Newton with dense solves: the first update (`solve`), or the converged state."""
    fixed = constrained(vmask)
    target = torch.zeros(m.nodes, 4, dtype=torch.float64)
    target[:, :3] = torch.from_numpy(np.asarray(inlet).reshape(-1, 3))
    target, state = target.cuda().reshape(-1), torch.from_numpy(start.copy()).cuda().reshape(-1)
    for _ in range(1 if kind == "solve" else 12):
        rhs, matrix = exact_assembly(m, state, start, dt, "matrix")
        rhs = torch.where(fixed, target - state, rhs)
        matrix[fixed] = 0.0
        matrix[fixed, fixed.nonzero()[:, 0]] = 1.0
        factors = torch.linalg.lu_factor(matrix)
        update = torch.linalg.lu_solve(*factors, rhs[:, None])
        update = (update + torch.linalg.lu_solve(*factors, rhs[:, None] - matrix @ update))[:, 0]
        if kind == "solve":
            return update.reshape(-1, 4)
        state = state + update
        if update.norm() <= 1e-13 * state.norm():
            break
    return state.reshape(-1, 4)


def exact_transport(case, seed, body):
    """Both matrices as dense ones, and a direct solve for every step."""
    m, n, c = body.mesh, body.mesh.nodes, TRANSPORT
    velocity = poiseuille(case, body, seed)
    mask, n0, nplus = api.resolve_transport_boundaries(body.labels, velocity, api.transport_params(**c))
    flow = torch.from_numpy(velocity).cuda()
    left = torch.zeros(n, 2, n, 2, dtype=torch.float64, device="cuda")
    mass, moved = (torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(2))
    dt = c["dt"]
    for el in slices(m, 400):
        value, grad, w = el.phi[:, :, 0], el.phi[:, :, 1:4], el.weight
        u = torch.einsum("eqa,eac->eqc", value, flow[el.nodes] * el.used[..., None])
        along = torch.einsum("eqc,eqca->eqa", u, grad)
        space = along.abs().sum(-1)
        tau = torch.where(space > 0, (space ** 2 + 4 / dt ** 2).rsqrt(), torch.zeros_like(space))
        test = value + tau[..., None] * along
        form = lambda a, b: torch.einsum("eq,eqa,eqb->eab", w, a, b)                    # noqa: E731
        stiff = torch.einsum("eq,eqca,eqcb->eab", w, grad, grad)
        gg = torch.einsum("eqca,eqcb->eqab", grad, grad)
        advect = form(test, along) * dt + dt * c["vplus"] * c["artificial_diffusion"] * torch.einsum(
            "eq,eqa,eqab->eab", w, test, gg)
        M, P = form(value, value), form(test, value)
        at = (el.nodes[:, :, None].expand(-1, -1, 64), el.nodes[:, None, :].expand(-1, 64, -1))
        view = left.permute(1, 3, 0, 2)
        for (i, f), block in {(0, 0): (1 + dt * (c["kplus"] + c["kminus"])) * M + dt * c["diffusion"] * stiff,
                              (0, 1): -c["detach_plus"] * dt * M, (1, 0): -c["kplus"] * dt * P,
                              (1, 1): (1 + dt * c["detach_plus"]) * P + advect}.items():
            view[i, f].index_put_(at, block, accumulate=True)
        mass.index_put_(at, M, accumulate=True)
        moved.index_put_(at, P, accumulate=True)
    fixed = torch.from_numpy(np.asarray(mask) != 0).cuda()
    given = torch.from_numpy(np.stack([n0, nplus], -1)).cuda()
    left[fixed] = 0.0
    node = fixed.nonzero()[:, 0]
    for k in range(2):
        left[node, k, node, k] = 1.0
    factors = torch.linalg.lu_factor(left.reshape(2 * n, 2 * n))
    state = torch.where(fixed[:, None], given, torch.zeros_like(given))
    for _ in range(case["steps"]):
        rhs = torch.stack([mass @ state[:, 0], moved @ state[:, 1]], -1)
        rhs = torch.where(fixed[:, None], given, rhs)
        state = torch.linalg.lu_solve(*factors, rhs.reshape(-1, 1)).reshape(-1, 2)
    return {"species": state.reshape(-1)}
