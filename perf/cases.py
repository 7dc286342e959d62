"""Performance cases: the calls a user of this library makes, timed through its public entry points.

Every case is a plain dict.  ``kind`` says which call it is:

- ``mltadd_host``: ``y <- beta y + alpha A x`` on host vectors (``FemMatrixFreeOperator.MltAddVector``), the call that
  replaces the reference's matrix-vector product in a host solver;
- ``mltadd``: the same product on device vectors (``mltadd_device``), the call of a solver that lives on the GPU;
- ``advance``: time steps of one run with the state on the device (``LeapFrogIterator.Advance``), with the norm and the
  receiver traces of every iterate when ``diag`` is set, by the order-2 or the order-4 scheme (``scheme``);
- ``sources``: many sources on one mesh advanced together, receivers recorded (``BatchLeapFrog.advance``);
- ``meshes``: runs on meshes of different size and order advanced together (``MeshBatch.advance``);
- ``adjoint``: the trace misfit and its gradient by wave speed (``adjoint.misfit`` and its backward).

Meshes are boxes of nx x ny x nz perturbed hexahedra (``mesh`` = ``random``: vertices moved by up to 5% of the cell
size; ``sin``: smooth displacement of 10%), the wave speed one value per element.  Fields start from a few smooth
waves, sources are Gaussian balls with a Ricker pulse.
"""
import math

import numpy as np
import torch

from montjoie_gb300.adjoint import AcousticAdjoint, misfit
from montjoie_gb300.leapfrog import BatchLeapFrog, LeapFrogIterator, MeshBatch
from montjoie_gb300.mesh import AcousticSetup, HexMesh
from montjoie_gb300.problem import AcousticProblem, geometry

# n_rec receivers per run with the order's (r+1)^3 interpolation weights each
RUN_RECEIVERS = 8
SHOT_RECEIVERS = 64


def listed():
    return [
        # the smallest call: one matrix-vector product on host vectors from a host solver's inner loop
        dict(name="mltadd host fp64 q2 6x5x4", kind="mltadd_host", precision="fp64", order=2, nx=6, ny=5, nz=4,
             mesh="random", alpha=1.0, beta=0.0),
        # a product inside a GPU-resident FP64 solver, ragged box, accumulating into y
        dict(name="mltadd fp64 q4 23x21x19", kind="mltadd", precision="fp64", order=4, nx=23, ny=21, nz=19,
             mesh="random", alpha=-0.7, beta=0.5),
        # one step at a time on a small mesh with diagnostics: a driver that looks at every iterate
        dict(name="step fp32 q4 12x12x12", kind="advance", precision="fp32", order=4, nx=12, ny=12, nz=12,
             mesh="random", scheme=2, steps=1, diag=True),
        # the plain method: 16^3 Q4, FP64, 200 steps, norm and traces
        dict(name="run fp64 q4 16x16x16", kind="advance", precision="fp64", order=4, nx=16, ny=16, nz=16,
             mesh="random", scheme=2, steps=200, diag=True),
        # the same method at scale: 64^3 Q4 in FP64
        dict(name="run fp64 q4 64x64x64", kind="advance", precision="fp64", order=4, nx=64, ny=64, nz=64,
             mesh="random", scheme=2, steps=10, diag=False),
        # high order in FP64 on an odd box
        dict(name="run fp64 q8 15x13x11", kind="advance", precision="fp64", order=8, nx=15, ny=13, nz=11,
             mesh="sin", scheme=2, steps=25, diag=False),
        # the headline workload: 64^3 Q4 in the FP32 form, norm and traces of every step
        dict(name="run fp32 q4 64x64x64", kind="advance", precision="fp32", order=4, nx=64, ny=64, nz=64,
             mesh="random", scheme=2, steps=40, diag=True),
        # high order on a curved mesh, FP32
        dict(name="run fp32 q8 32x32x32", kind="advance", precision="fp32", order=8, nx=32, ny=32, nz=32,
             mesh="sin", scheme=2, steps=30, diag=False),
        # the order-4 scheme, FP32, low order elements on a ragged box
        dict(name="order4 fp32 q3 45x37x41", kind="advance", precision="fp32", order=3, nx=45, ny=37, nz=41,
             mesh="random", scheme=4, steps=40, diag=False),
        # a survey: 64 shots on one 32^3 Q4 mesh, 64 receivers
        dict(name="shots fp32 q4 32x32x32 64", kind="sources", order=4, nx=32, ny=32, nz=32, mesh="random",
             shots=64, steps=12),
        # an ensemble of meshes of uneven size and order
        dict(name="ensemble fp32 12 meshes", kind="meshes", meshes=12, lo=8, hi=22, mesh="random", steps=40),
        # inversion: misfit and gradient of 16 shots x 64 receivers
        dict(name="gradient q4 16x16x16 16", kind="adjoint", order=4, nx=16, ny=16, nz=16, mesh="random",
             shots=16, steps=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# dofs of the largest runs listed above, a little less (a drawn case costs no more than they do)
_MOST_DOFS = 16.0e6


def _box(rng, order, most_dofs, least=2):
    """An uneven box whose dofs are spread over the logarithm of [small, most_dofs]."""
    dofs = math.exp(rng.uniform(math.log(400.0), math.log(most_dofs)))
    side = max(1.0 * least, dofs ** (1.0 / 3.0) / order)
    return [max(least, int(side * rng.uniform(0.8, 1.1))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["mltadd_host", "mltadd", "advance", "advance", "advance", "advance", "sources", "meshes",
                       "adjoint"])
    order = rng.choice([1, 2, 3, 4, 4, 4, 5, 6, 7, 8])
    mesh = rng.choice(["random", "sin"])
    if kind in ("mltadd_host", "mltadd"):
        nx, ny, nz = _box(rng, order, 4.0e5 if kind == "mltadd_host" else 6.0e6)
        return dict(kind=kind, precision=rng.choice(["fp64", "fp32"]), order=order, nx=nx, ny=ny, nz=nz, mesh=mesh,
                    alpha=round(rng.uniform(-2.0, 2.0), 3), beta=rng.choice([0.0, 1.0, round(rng.uniform(-1, 1), 3)]))
    if kind == "advance":
        precision = rng.choice(["fp64", "fp32"])
        scheme = rng.choice([2, 2, 2, 4])
        nx, ny, nz = _box(rng, order, _MOST_DOFS / (4 if precision == "fp64" and scheme == 4 else 1))
        dofs = order ** 3 * nx * ny * nz
        most = max(1, min(200, int((1.5e8 if precision == "fp64" else 6.0e8) / (scheme / 2) / dofs)))
        return dict(kind=kind, precision=precision, order=order, nx=nx, ny=ny, nz=nz, mesh=mesh, scheme=scheme,
                    steps=_log_int(rng, 1, most), diag=rng.random() < 0.5)
    if kind == "meshes":
        hi = _log_int(rng, 6, 20)
        return dict(kind=kind, meshes=rng.randint(2, 12), lo=max(2, hi // 3), hi=hi, mesh=mesh,
                    steps=_log_int(rng, 1, 40))
    shots = rng.choice([1, 3, 8, 13, 16, 24, 32, 64])
    nx, ny, nz = _box(rng, order, (1.2e8 if kind == "sources" else 4.0e6) / max(shots, 8))
    if kind == "sources":
        return dict(kind=kind, order=order, nx=nx, ny=ny, nz=nz, mesh=mesh, shots=shots, steps=_log_int(rng, 1, 12))
    return dict(kind=kind, order=order, nx=nx, ny=ny, nz=nz, mesh=mesh, shots=shots, steps=rng.randint(30, 100))


# ---------------------------------------------------------------- the mesh and the media (numpy, from the seed alone)

_CORNERS = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])


def _mesh(nx, ny, nz, kind, rng, c_lo=1.0, c_hi=3.0):
    """(HexMesh, cell size): a box of unit-aspect cells, its longest side 1, elements and vertices in lexicographic
    order (x fastest), wave speed U[c_lo, c_hi] per element."""
    h = 1.0 / max(nx, ny, nz)
    iz, iy, ix = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    idx = np.stack([ix, iy, iz], axis=-1).reshape(-1, 3)
    verts = idx * h
    free = (idx > 0) & (idx < np.array([nx, ny, nz]))
    if kind == "random":
        verts = verts + free * rng.uniform(-0.05 * h, 0.05 * h, size=verts.shape)
    else:
        verts = verts + free * (0.1 * h * np.prod(np.sin(2 * np.pi * verts), axis=1, keepdims=True))
    ez, ey, ex = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    hexes = np.stack([((ez + c[2]) * (ny + 1) + ey + c[1]) * (nx + 1) + ex + c[0] for c in _CORNERS], axis=1)
    ne = hexes.shape[0]
    m = HexMesh(verts=verts, hexes=hexes.astype(np.int32), elem_ref=np.arange(1, ne + 1, dtype=np.int32),
                media_c=rng.uniform(c_lo, c_hi, size=ne), bfaces=np.zeros((0, 4), dtype=np.int32), n=0)
    return m, h


def _lobatto(r):
    """Gauss-Lobatto points on [0, 1], weights and G[a, b] = phi_a'(x_b), from the Legendre polynomial of degree r."""
    c = np.zeros(r + 1)
    c[r] = 1.0
    inner = np.sort(np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c)).real) if r > 1 else np.zeros(0)
    d1, d2, d3 = (np.polynomial.legendre.legder(c, k) if r >= k else np.zeros(1) for k in (1, 2, 3))
    val = np.polynomial.legendre.legval
    for _ in range(3 if r > 1 else 0):  # Newton steps on P_r'
        f, g = val(inner, d1), val(inner, d2)
        inner = inner - f / g
    x = np.concatenate([[-1.0], inner, [1.0]])
    w = 1.0 / (r * (r + 1) * val(x, c) ** 2)
    x = 0.5 * (x + 1.0)
    diff = x[:, None] - x[None, :] + np.eye(r + 1)
    b = 1.0 / diff.prod(axis=1)
    G = b[:, None] / b[None, :] / (diff.T - np.eye(r + 1) + np.eye(r + 1))
    np.fill_diagonal(G, 0.0)
    np.fill_diagonal(G, -G.sum(axis=0))
    return x, w, G


def _local_points(r):
    """(i, j, k) of every local node in the library's element order: vertices, edges, faces, interior."""
    edges = [(0, 1), (1, 2), (3, 2), (0, 3), (0, 4), (1, 5), (2, 6), (3, 7), (4, 5), (5, 6), (7, 6), (4, 7)]
    pts = [r * c for c in _CORNERS]
    for a, b in edges:
        pts += [_CORNERS[a] * r + s * (_CORNERS[b] - _CORNERS[a]) for s in range(1, r)]
    inner = range(1, r)
    for axis, side in ((0, 0), (1, 0), (2, 0), (2, r), (1, r), (0, r)):
        pts += [np.insert([p, q], axis, side) for p in inner for q in inner]
    pts += [np.array([i, j, k]) for i in inner for j in inner for k in inner]
    return np.array(pts)


def _block_order(r):
    """Where the numbering of a mesh in lexicographic order meets each local node of an element: first the place
    (x fastest) at which its vertex, edge, face or interior is met, then its place within that block (x fastest in
    the interior, x or else y slowest on a face)."""
    n = r + 1
    pts = _local_points(r)
    sort = np.where(pts == 0, 0, np.where(pts == r, 2, 1))  # low end, inside, high end of each axis
    place = (pts[:, 2] * n + pts[:, 1]) * n + pts[:, 0]
    entity = (sort[:, 2] * 3 + sort[:, 1]) * 3 + sort[:, 0]
    met = np.array([place[entity == t].min() for t in entity])
    on_face = (sort == 1).sum(1) == 2
    return met * n ** 3 + np.where(on_face, (pts[:, 0] * n + pts[:, 1]) * n + pts[:, 2], place)


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, case.get("order", 0), case.get("nx", 0), case.get("steps", 0)])


def _smooth(rng):
    """A few waves: (wave vectors, phases, amplitudes)."""
    return rng.uniform(-6.0, 6.0, (4, 3)), rng.uniform(0.0, 6.0, 4), rng.uniform(0.2, 1.0, 4)


def _field(wave, x):
    k, ph, a = (torch.as_tensor(v, device=x.device) for v in wave)
    return (torch.sin(x @ k.T + ph) * a).sum(-1)


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _points(r, mesh):
    """Physical points (ne, Q, 3) in local order, on the device."""
    x = torch.as_tensor(_lobatto(r)[0], device=_device())
    xi = x[torch.as_tensor(_local_points(r), device=_device())]
    v = torch.as_tensor(mesh.verts[mesh.hexes], device=_device())
    c = torch.as_tensor(_CORNERS, device=_device(), dtype=torch.float64)
    shape = torch.prod(c[None] * xi[:, None] + (1 - c[None]) * (1 - xi[:, None]), dim=2)
    return torch.einsum("qc,ecd->eqd", shape, v)


def _dof_field(wave, r, mesh, nodle, n_dof):
    u = torch.zeros(n_dof, dtype=torch.float64, device=_device())
    nod = torch.as_tensor(np.ascontiguousarray(nodle), device=_device()).long().reshape(-1)
    # one value per dof whatever the element it is taken from: the last bits of a point's position differ between
    # its elements, so each dof takes the value of its first element
    first = torch.full((n_dof,), nod.numel(), dtype=torch.long, device=_device())
    first.scatter_reduce_(0, nod, torch.arange(nod.numel(), device=_device()), reduce="amin")
    x = _points(r, mesh).reshape(-1, 3)
    u[:] = _field(wave, x[first])
    return u


def _time_step(r, h, c_max, scheme):
    x = _lobatto(r)[0]
    return 0.3 * (x[1] - x[0]) * h / c_max * (1.5 if scheme == 4 else 1.0)


def _ricker(dt, steps):
    """Pulse at (n+1) dt, n = 0..steps-1, and its second time derivative; the peak lies inside the first steps."""
    f0 = 1.0 / (24.0 * dt)
    a = np.pi * f0 * ((np.arange(max(steps, 64)) + 1) * dt - 12.0 * dt)
    g = np.exp(-a * a)
    return (1 - 2 * a * a) * g, -(8 * a ** 4 - 24 * a * a + 6) * g * (np.pi * f0) ** 2


def _receivers(rng, r, n_elt, n_rec):
    """Receivers inside elements: (element, weights of its local nodes)."""
    x = _lobatto(r)[0]
    el = rng.integers(0, n_elt, n_rec)
    xi = rng.uniform(0.05, 0.95, (n_rec, 3))
    L = np.ones((n_rec, 3, r + 1))
    for a in range(r + 1):
        for b in range(r + 1):
            if a != b:
                L[:, :, a] *= (xi - x[b]) / (x[a] - x[b])
    p = _local_points(r)
    return el, L[:, 0, p[:, 0]] * L[:, 1, p[:, 1]] * L[:, 2, p[:, 2]]


def _shot_points(rng, case, h):
    box = np.array([case["nx"], case["ny"], case["nz"]]) * h
    return rng.uniform(0.25, 0.75, (case["shots"], 3)) * box


def _setup(case, seed):
    """Mesh, media and every random choice of a case, in one order, for prepare() and exact() alike."""
    rng = _rng(case, seed)
    r = case["order"]
    mesh, h = _mesh(case["nx"], case["ny"], case["nz"], case["mesh"], rng)
    scheme = case.get("scheme", 2)
    s = dict(r=r, mesh=mesh, h=h, dt=_time_step(r, h, 3.0, scheme), wave=_smooth(rng), wave2=_smooth(rng),
             center=np.array([case["nx"], case["ny"], case["nz"]]) * h * rng.uniform(0.4, 0.6, 3), radius=2.5 * h)
    n_rec = SHOT_RECEIVERS if case["kind"] in ("sources", "adjoint") else RUN_RECEIVERS
    s["rec_el"], s["rec_w"] = _receivers(rng, r, mesh.n_elt, n_rec)
    if "shots" in case:
        s["points"] = _shot_points(rng, case, h)
    s["c_true"] = mesh.media_c * (1.0 + 0.05 * rng.uniform(-1, 1, mesh.n_elt))
    return s


# ---------------------------------------------------------------- what a user's program holds before the call


class _Buffer:
    """A device buffer of an integrator for torch, without a copy; a tensor made from it keeps the integrator."""

    def __init__(self, owner, ptr, n, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": np.dtype(dtype).str, "data": (ptr, False),
                                         "version": 3, "strides": None}


def _views(lf):
    a, b, _ = lf.device_state()
    return {p: torch.as_tensor(_Buffer(lf, p, lf.op.n_dof, lf.op.dtype), device="cuda") for p in (a, b)}


def _problem(s):
    return AcousticProblem(s["mesh"], AcousticSetup(order=s["r"], src_center=tuple(s["center"]),
                                                    src_radius=s["radius"]), defer_time=True)


def _integrator(s, pb, op, case):
    p, p2 = _ricker(s["dt"], 0)
    diag = case.get("diag", False)
    lf = LeapFrogIterator(op, s["dt"], pb.mass, None, pb.src_idx, pb.src_val, p, pb.norm_weight if diag else None,
                          pb.nodle[s["rec_el"]] if diag else None, s["rec_w"] if diag else None,
                          time_order=case.get("scheme", 2), pulse_d2=p2 if case.get("scheme", 2) == 4 else None)
    lf.SetInitialConditionS(_dof_field(s["wave"], s["r"], s["mesh"], pb.nodle, pb.n_dof).cpu().numpy())
    return lf


def _shots(s, op):
    idx, rhs, val = [], [], []
    for k, c in enumerate(s["points"]):
        i, v = op.gaussian_source(c, s["radius"])
        idx.append(i)
        val.append(v)
        rhs.append(np.full(i.size, k, dtype=np.int32))
    return np.concatenate(idx), np.concatenate(rhs), np.concatenate(val)


def _ensemble_shapes(case):
    """(order, nx, ny, nz) of every run: orders 2, 3, 4, 6 and 8 in turn, sides spread over [lo, hi] at order 4 (the
    others get about as many dofs)."""
    out = []
    for k in range(case["meshes"]):
        order = [2, 3, 4, 6, 8][k % 5]
        side = case["lo"] + (case["hi"] - case["lo"]) * ((0.5 + 0.618034 * k) % 1.0)
        side = max(2, round(side * 4 / max(order, 3)))
        out.append((order, side, side, max(2, side - k % 3)))
    return out


def _ensemble(case, seed):
    """The runs of a mesh ensemble as (case, seed) of their own."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, case["meshes"]])
    return [(dict(kind="advance", precision="fp32", order=order, nx=nx, ny=ny, nz=nz, mesh=case["mesh"], scheme=2,
                  steps=case["steps"], diag=False), int(rng.integers(1 << 30)))
            for order, nx, ny, nz in _ensemble_shapes(case)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "meshes":
        runs, ops = [], []
        for sub, sub_seed in _ensemble(case, seed):
            s = _setup(sub, sub_seed)
            pb = _problem(s)
            ops.append(pb.operator("fp32"))
            runs.append(_integrator(s, pb, ops[-1], sub))
        return dict(case=case, ops=ops, runs=runs, batch=MeshBatch(runs), views=[_views(lf) for lf in runs])
    s = _setup(case, seed)
    if kind == "adjoint":
        one = HexMesh(verts=s["mesh"].verts, hexes=s["mesh"].hexes, elem_ref=np.ones(s["mesh"].n_elt, dtype=np.int32),
                      media_c=np.ones(1), bfaces=s["mesh"].bfaces, n=0)
        pb = _problem(dict(s, mesh=one))
        factors, _, _ = geometry(s["r"], pb.verts_e, pb.mu, want_positions=False)
        op = pb.operator("fp32")
        idx, rhs, val = _shots(s, op)
        op.close()
        model = AcousticAdjoint(s["r"], pb.nodle, factors, pb.n_dof, pb.mass, s["dt"], case["steps"], case["shots"],
                                idx, rhs, val, _ricker(s["dt"], case["steps"])[0], pb.nodle[s["rec_el"]], s["rec_w"])
        data = model.forward(s["c_true"])
        c = torch.tensor(s["mesh"].media_c, dtype=torch.float64, device="cuda", requires_grad=True)
        return dict(case=case, model=model, data=data, c=c)
    pb = _problem(s)
    if kind == "sources":
        op = pb.operator("fp32")
        idx, rhs, val = _shots(s, op)
        batch = BatchLeapFrog(op, s["dt"], case["shots"], pb.mass, None, idx, rhs, val, _ricker(s["dt"], 0)[0],
                              pb.nodle[s["rec_el"]], s["rec_w"])
        u0 = _dof_field(s["wave"], s["r"], s["mesh"], pb.nodle, pb.n_dof)
        gain = torch.linspace(0.5, 1.5, case["shots"], dtype=torch.float64, device=u0.device)
        batch.init((u0[:, None] * gain).cpu().numpy())
        return dict(case=case, op=op, batch=batch)
    op = pb.operator(case["precision"])
    if kind == "advance":
        lf = _integrator(s, pb, op, case)
        pb.close()
        return dict(case=case, op=op, lf=lf, views=_views(lf))
    x = _dof_field(s["wave"], s["r"], s["mesh"], pb.nodle, pb.n_dof)
    y = _dof_field(s["wave2"], s["r"], s["mesh"], pb.nodle, pb.n_dof)
    pb.close()
    if kind == "mltadd_host":
        return dict(case=case, op=op, x=x.cpu().numpy(), y=y.cpu().numpy())
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    return dict(case=case, op=op, x=x.to(dtype), y=y.to(dtype))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mltadd_host":
        state["op"].MltAddVector(case["alpha"], state["x"], case["beta"], state["y"])
        return state["y"]
    if kind == "mltadd":
        state["op"].mltadd_device(case["alpha"], state["x"].data_ptr(), case["beta"], state["y"].data_ptr(),
                                  torch.cuda.current_stream().cuda_stream)
        return state["y"]
    if kind == "advance":
        norms, traces = state["lf"].Advance(case["steps"])
        a, b, _ = state["lf"].device_state()
        out = [state["views"][a], state["views"][b]]
        return out + [norms, traces] if case["diag"] else out
    if kind == "sources":
        return state["batch"].advance(case["steps"], traces=True)
    if kind == "meshes":
        state["batch"].advance(case["steps"])
        return [[v[p] for p in lf.device_state()[:2]] for lf, v in zip(state["runs"], state["views"])]
    state["c"].grad = None
    loss = misfit(state["c"], state["model"], state["data"])
    loss.backward()
    return [loss.detach(), state["c"].grad]


# ---------------------------------------------------------------- floors


def _sizes(case):
    r = case["order"]
    ne = case["nx"] * case["ny"] * case["nz"]
    return r, ne, (r + 1) ** 3, (case["nx"] * r + 1) * (case["ny"] * r + 1) * (case["nz"] * r + 1)


def work(case):
    """Bytes and operations of one pass: per stiffness product the six factors and the connectivity of every point
    and the vector; per step the two states read, one written and the mass; six contractions of n points and the
    3 x 3 factors per point."""
    kind = case["kind"]
    if kind == "meshes":
        total = {"bytes": 0.0, "flops": 0.0}
        for sub, _ in _ensemble(case, 0):
            w = work(sub)
            total = {q: total[q] + w[q] for q in total}
        return total
    r, ne, q, nd = _sizes(case)
    sz = 4 if case.get("precision", "fp32") == "fp32" else 8
    per_point = 2.0 * (6 * (r + 1) + 9)
    product = ne * q * (6 * sz + 4.0)
    if kind in ("mltadd", "mltadd_host"):
        vec = nd * (8 if kind == "mltadd_host" else sz) * (2 + (case["beta"] != 0.0))
        return {"bytes": product + vec, "flops": ne * q * per_point}
    if kind == "advance":
        k = case["steps"] * (case["scheme"] // 2)
        return {"bytes": k * product + case["steps"] * nd * 4.0 * sz, "flops": k * (ne * q * per_point + 4.0 * nd)}
    runs = case["shots"]
    steps = case["steps"] * (1 if kind == "sources" else 2)
    return {"bytes": steps * (product + nd * 4.0 + nd * runs * 12.0), "flops": steps * runs * (ne * q * per_point + 4.0 * nd)}


# ---------------------------------------------------------------- the same results in 64 bits


class _Plain:
    """The stiffness product, mass and sources of a box mesh in FP64 tensors."""

    def __init__(self, s, case, mu):
        r, mesh, dev = s["r"], s["mesh"], _device()
        n = r + 1
        x, w, G = (torch.as_tensor(v, device=dev) for v in _lobatto(r))
        self.n, self.G = n, G
        v = torch.as_tensor(mesh.verts[mesh.hexes], device=dev).reshape(-1, 8, 3)
        # [e, i, j, k] grids: trilinear map and its derivative
        lo, hi = 1 - x, x
        one = torch.ones_like(x)
        J = [[0.0] * 3 for _ in range(3)]
        X = 0.0
        for c, (a, b, g) in enumerate(_CORNERS):
            A, B, C = (hi if a else lo), (hi if b else lo), (hi if g else lo)
            dA, dB, dC = (one if a else -one), (one if b else -one), (one if g else -one)
            N = [torch.einsum("i,j,k->ijk", *t) for t in ((A, B, C), (dA, B, C), (A, dB, C), (A, B, dC))]
            for d in range(3):
                vd = v[:, c, d][:, None, None, None]
                for e in range(3):
                    J[d][e] = J[d][e] + vd * N[1 + e]
            X = X + v[:, c][:, None, None, None, :] * N[0][None, ..., None]
        cof = [[J[(d + 1) % 3][(e + 1) % 3] * J[(d + 2) % 3][(e + 2) % 3]
                - J[(d + 1) % 3][(e + 2) % 3] * J[(d + 2) % 3][(e + 1) % 3] for e in range(3)] for d in range(3)]
        det = sum(J[0][e] * cof[0][e] for e in range(3))
        w3 = torch.einsum("i,j,k->ijk", w, w, w)
        self.jw = det * w3
        scale = w3 / det * torch.as_tensor(mu, device=dev)[:, None, None, None]
        self.B = {(a, b): scale * sum(cof[d][a] * cof[d][b] for d in range(3)) for a in range(3) for b in range(a, 3)}
        self.X = X
        # dofs numbered as the elements first touch them, each vertex, edge, face and interior one block (_block_order)
        lat = torch.as_tensor(_local_points(r), device=dev)
        ex, ey, ez = case["nx"], case["ny"], case["nz"]
        e = torch.arange(ex * ey * ez, device=dev)
        e3 = torch.stack([e % ex, (e // ex) % ey, e // (ex * ey)], 1)
        p = e3[:, None, :] * r + lat[None]
        node = ((p[..., 2] * (ey * r + 1) + p[..., 1]) * (ex * r + 1) + p[..., 0]).reshape(-1)
        self.n_dof = (ex * r + 1) * (ey * r + 1) * (ez * r + 1)
        met = (e[:, None] * n ** 6 + torch.as_tensor(_block_order(r), device=dev)[None]).reshape(-1)
        first = torch.full((self.n_dof,), 1 << 62, dtype=torch.long, device=dev)
        first.scatter_reduce_(0, node, met, reduce="amin")
        rank = torch.empty_like(first)
        rank[torch.argsort(first)] = torch.arange(self.n_dof, device=dev)
        self.nodle = rank[node].reshape(-1, n ** 3)
        grid = torch.empty((n, n, n), dtype=torch.long, device=dev)
        grid[lat[:, 0], lat[:, 1], lat[:, 2]] = torch.arange(n ** 3, device=dev)
        self.nod = self.nodle[:, grid.reshape(-1)].reshape(-1, n, n, n)
        self.D = self.gather(self.jw)

    def gather(self, y):
        out = torch.zeros(y.shape[:-4] + (self.n_dof,), dtype=torch.float64, device=y.device)
        return out.index_add_(-1, self.nod.reshape(-1), y.reshape(y.shape[:-4] + (-1,)))

    def parts(self, u):
        """Element-local A u, [..., e, i, j, k]."""
        G, B = self.G, self.B
        ul = u[..., self.nod]
        g = [torch.einsum("al,...ajk->...ljk", G, ul), torch.einsum("am,...iak->...imk", G, ul),
             torch.einsum("ap,...ija->...ijp", G, ul)]
        f = [sum(B[min(a, b), max(a, b)] * g[b] for b in range(3)) for a in range(3)]
        return (torch.einsum("ia,...ajk->...ijk", G, f[0]) + torch.einsum("ja,...iak->...ijk", G, f[1])
                + torch.einsum("ka,...ija->...ijk", G, f[2]))

    def apply(self, u):
        return self.gather(self.parts(u))

    def ball(self, center, radius):
        alpha = -math.log(1e-6) / (radius * radius)
        d2 = ((self.X - torch.as_tensor(center, device=self.X.device)) ** 2).sum(-1)
        f = self.jw * math.sqrt(alpha / math.pi) * torch.exp(-alpha * d2)
        return self.gather(torch.where(d2.sqrt() < radius, f, torch.zeros_like(f)))

    def traces(self, s, u):
        """Receiver values of u: [..., n_rec]."""
        idx = self.nodle[torch.as_tensor(s["rec_el"], device=u.device)]
        return (u[..., idx] * torch.as_tensor(s["rec_w"], device=u.device)).sum(-1)


def _leapfrog(P, dt, u0, F, pulse, pulse2, steps, scheme, see=None):
    """U^steps and U^(steps+1); see(k, U^k) is called for k = 0..steps-1."""
    D = P.D
    d2 = -P.apply(u0) / D
    prev = u0
    if scheme == 4:
        d4 = -P.apply(d2) / D
        cur = u0 + dt * dt * (d2 / 2 + dt * dt * d4 / 24)
    else:
        cur = u0 + 0.5 * dt * dt * d2
    for k in range(steps):
        if see is not None:
            see(k, prev)
        p = pulse[k] if k < len(pulse) else 0.0
        p2 = pulse2[k] if k < len(pulse2) else 0.0
        w = dt * dt * (p * F - P.apply(cur))
        new = 2 * cur - prev + w / D
        if scheme == 4:
            new = new + dt * dt / 12 * (dt * dt * p2 * F - P.apply(w / D)) / D
        prev, cur = cur, new
    return prev, cur


def exact(case, seed):
    kind = case["kind"]
    if kind == "meshes":
        out = []
        for sub, sub_seed in _ensemble(case, seed):
            out.append(exact(sub, sub_seed))
        return out
    s = _setup(case, seed)
    steps = case.get("steps", 1)
    if kind == "adjoint":
        return _exact_gradient(case, s)
    P = _Plain(s, case, s["mesh"].media_c ** 2)
    u0 = _dof_field(s["wave"], s["r"], s["mesh"], P.nodle.cpu().numpy(), P.n_dof)
    pulse, pulse2 = _ricker(s["dt"], 0)
    if kind in ("mltadd", "mltadd_host"):
        y = _dof_field(s["wave2"], s["r"], s["mesh"], P.nodle.cpu().numpy(), P.n_dof)
        out = case["beta"] * y + case["alpha"] * P.apply(u0)
        return out.cpu().numpy() if kind == "mltadd_host" else out
    if kind == "advance":
        norms, traces = [], []

        def see(k, u):
            if case["diag"]:
                norms.append((P.D * u * u).sum())
                traces.append(P.traces(s, u))

        a, b = _leapfrog(P, s["dt"], u0, P.ball(s["center"], s["radius"]), pulse, pulse2, steps, case["scheme"], see)
        return [a, b] + ([torch.stack(norms), torch.stack(traces, 1)] if case["diag"] else [])
    gain = torch.linspace(0.5, 1.5, case["shots"], dtype=torch.float64, device=u0.device)
    out = []
    group = max(1, int(6e8 / (P.nod.numel() * 8 * 4)))
    for at in range(0, case["shots"], group):
        F = torch.stack([P.ball(c, s["radius"]) for c in s["points"][at:at + group]])
        rows = []
        _leapfrog(P, s["dt"], gain[at:at + group, None] * u0, F, pulse, pulse2, steps, 2,
                  lambda k, u: rows.append(P.traces(s, u)))
        out.append(torch.stack(rows, 2))
    return torch.cat(out, 0).permute(1, 0, 2).contiguous()


def _exact_gradient(case, s):
    """Loss and gradient by the discrete adjoint of the leap-frog, in FP64: with the constraint
    D (U^m - 2 U^(m-1) + U^(m-2)) + dt^2 (A U^(m-1) - p F) = 0, dJ/dc_e = sum_m lambda^m . dt^2 (2 / c_e) A_e U^(m-1)."""
    dt, N, c = s["dt"], case["steps"], s["mesh"].media_c
    pulse = _ricker(dt, N)[0]

    def forward(c):
        P = _Plain(s, case, c ** 2)
        F = torch.stack([P.ball(x, s["radius"]) for x in s["points"]])
        states = [torch.zeros_like(F), torch.zeros_like(F)]
        for k in range(N - 1):
            states.append(2 * states[-1] - states[-2] + dt * dt / P.D * (pulse[k] * F - P.apply(states[-1])))
        return P, states, torch.stack([P.traces(s, u) for u in states], 2)

    data = forward(s["c_true"])[2]
    P, U, tr = forward(c)
    res = tr - data
    idx = P.nodle[torch.as_tensor(s["rec_el"], device=res.device)]
    w = torch.as_tensor(s["rec_w"], device=res.device)
    grad = torch.zeros(len(c), dtype=torch.float64, device=res.device)
    lam1, lam2 = torch.zeros_like(U[0]), torch.zeros_like(U[0])  # lambda^(m+1), lambda^(m+2)
    parts = torch.zeros(U[0].shape[:1] + P.nod.shape, dtype=torch.float64, device=res.device)  # A_e lambda^(m+1)
    for m in range(N, 1, -1):
        g = torch.zeros_like(lam1)
        g.index_add_(-1, idx.reshape(-1), (res[:, :, m, None] * w).reshape(res.shape[0], -1))
        lam = 2 * lam1 - lam2 - (dt * dt * P.gather(parts) + g) / P.D
        parts = P.parts(lam)
        grad += (parts * U[m - 1][..., P.nod]).sum((0, 2, 3, 4))
        lam1, lam2 = lam, lam1
    grad = grad * 2 * dt * dt / torch.as_tensor(c, device=res.device)
    return [0.5 * (res * res).sum(), grad]
