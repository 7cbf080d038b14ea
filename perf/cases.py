"""Workloads of the explicit time step, from the smallest calls to the largest
meshes, through the Python binding and the C ABI's device pointers.

A case is a dict of plain values:
  element    "tet4" (each cell of a box split into 6), "hex8" or "tri6" (each
             cell of a square split into 2)
  nx, ny, nz cells along each axis (nz is 0 for triangles)
  law        "elastic", "neohookean" or "plastic"
  precision  "fp64", "mixed" or "fp64_fast"
  points     quadrature rule of triangles: 3 or 6 points (0 otherwise)
  distort    the inner nodes are displaced, so no element is a parallelepiped
  flow       how a program drives the steps
             "run"     solveStep(steps), the state read where it lies
             "watch"   solveStep(1) and getDisplacement(), steps times: a
                       script that looks at every step on the host
             "stream"  every step uploads its external force from pinned memory
                       and reads the displacement back, four reads in flight
             "batch"   `count` independent cubes of nx..ny cells per edge
                       advanced together by solveStep(steps)
  steps      time steps of one pass
  count      cubes of a batch (1 otherwise)
"""
import ctypes
import math
import random

import numpy as np
import torch

import akantu2_b200 as akb

_DISPLACEMENT, _VELOCITY, _ACCELERATION = 0, 1, 2
_RHO, _E, _NU, _SIGMA_Y, _HARDENING = 1.0, 1.0, 0.3, 1e-3, 0.1
_TYPES = {"tet4": "_tetrahedron_4", "hex8": "_hexahedron_8", "tri6": "_triangle_6"}
_LAWS = {"elastic": "elastic", "neohookean": "neohookean",
         "plastic": "plastic_linear_isotropic_hardening"}
_NODES = {"tet4": 4, "hex8": 8, "tri6": 6}
_CELL_ELEMENTS = {"tet4": 6, "hex8": 1, "tri6": 2}
# stable time step x celerity / cell edge of the regular meshes below: twice
# the inradius of the tetrahedra, the edge of the hexahedra, the inradius of
# the corner triangles of the quadratic triangles
_STABLE = {"tet4": 0.41, "hex8": 1.0, "tri6": 0.29}
_RAMP_SPEED, _RAMP_STEPS = 1e-3, 5000


def _case(name, element, n, law, precision, steps, flow="run", points=0, distort=False, count=1):
    case = {"element": element, "nx": n[0], "ny": n[1], "nz": n[2], "law": law,
            "precision": precision, "steps": steps, "flow": flow, "points": points,
            "distort": distort, "count": count}
    return dict(case, name=name) if name else case


def listed():
    return [
        # a script that steps a small model and looks at the result every time
        _case("watch tet4 8^3 fp64", "tet4", (8, 8, 8), "elastic", "fp64", 1, flow="watch"),
        # a small parameter study: one graph of steps, bound by launches
        _case("run tet4 8^3 mixed", "tet4", (8, 8, 8), "elastic", "mixed", 100),
        # the 48,000-tetrahedron cube in the reference's own precision
        _case("run tet4 20^3 fp64", "tet4", (20, 20, 20), "elastic", "fp64", 100),
        # an ordinary part meshed with tetrahedra of odd counts, large strains,
        # a step count that is not a whole number of graphs
        _case("run tet4 61x47x53 neo", "tet4", (61, 47, 53), "neohookean", "mixed", 130),
        # the large hexahedral box
        _case("run hex8 128^3 neo", "hex8", (128, 128, 128), "neohookean", "mixed", 100),
        # the same law in the reference's precision and in its fast form
        _case("run hex8 56^3 neo fp64", "hex8", (56, 56, 56), "neohookean", "fp64", 100),
        _case("run hex8 72^3 neo fast", "hex8", (72, 72, 72), "neohookean", "fp64_fast", 100),
        # a swept mesh without any parallelepiped
        _case("run hex8 57x43x39 bent", "hex8", (57, 43, 39), "elastic", "mixed", 100,
              distort=True),
        # the plane-strain plastic square with its pulled edge, both rules
        _case("run tri6 512^2 plastic", "tri6", (512, 512, 0), "plastic", "mixed", 100, points=3),
        _case("run tri6 181x97 fp64", "tri6", (181, 97, 0), "plastic", "fp64", 100, points=6),
        # many independent cubes in one model
        _case("batch tet4 64 cubes", "tet4", (8, 32, 0), "elastic", "mixed", 100, flow="batch",
              count=64),
        # coupled to a program on the host: forces in, displacements out
        _case("stream hex8 64^3", "hex8", (64, 64, 64), "neohookean", "mixed", 20, flow="stream"),
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("tet4", "tet4", "hex8", "hex8", "tri6", "batch", "watch", "stream"))
    if kind == "batch":
        hi = span(10, 32)
        return _case(None, "tet4", (rng.randint(6, hi - 2), hi, 0),
                     rng.choice(("elastic", "neohookean")), rng.choice(("mixed", "mixed", "fp64")),
                     100, flow="batch", count=span(4, 64))
    if kind in ("watch", "stream"):
        n = span(6, 40)
        return _case(None, rng.choice(("tet4", "hex8")), (n, rng.randint(n, n + 5), n + 1),
                     rng.choice(("elastic", "neohookean")), rng.choice(("mixed", "fp64")),
                     rng.randint(1, 20), flow=kind)
    steps = rng.choice((40, 100, 100, 130, 200))
    if kind == "tri6":
        n = span(24, 440)
        return _case(None, "tri6", (n, rng.randint(max(8, n // 2), n), 0), "plastic",
                     rng.choice(("mixed", "fp64")), steps, points=rng.choice((3, 6)))
    precision = rng.choice(("mixed", "mixed", "fp64"))
    if kind == "tet4":
        n = span(6, 60)
        return _case(None, "tet4", (n, rng.randint(max(3, n // 2), n), rng.randint(max(3, n // 2), n)),
                     rng.choice(("elastic", "elastic", "neohookean")), precision, steps)
    n = span(6, 56 if precision == "fp64" else 100)
    return _case(None, "hex8", (n, rng.randint(max(3, n // 2), n), rng.randint(max(3, n // 2), n)),
                 rng.choice(("elastic", "neohookean", "neohookean")), precision, steps,
                 distort=rng.random() < 0.25)


# -- meshes, states and materials ---------------------------------------------------

def _cubes(case, seed):
    """(cells, E, nu) of each cube of a batch; the cells do not depend on the
    inputs' seed, so every pass of a case does the same work"""
    cells = random.Random(case["count"] * 1009 + case["nx"] * 31 + case["ny"])
    value = random.Random(seed)
    return [(cells.randint(case["nx"], case["ny"]), 2.0 ** value.uniform(-1.0, 1.0),
             value.uniform(0.2, 0.4)) for _ in range(case["count"])]


def _grid(cells):
    """points of a grid, x fastest; the longest edge has length 1"""
    axes = [np.arange(c + 1) / max(cells) for c in cells]
    mesh = np.meshgrid(*reversed(axes), indexing="ij")
    return np.stack([m.ravel() for m in reversed(mesh)], axis=1)


def _mesh(element, cells, distort=False):
    """nodes and connectivity of a box of cells[0] x cells[1] (x cells[2])"""
    if element == "tri6":
        cx, cy = cells
        mx = 2 * cx + 1
        nodes = _grid((2 * cx, 2 * cy))
        j, i = np.meshgrid(np.arange(cy), np.arange(cx), indexing="ij")
        at = lambda a, b: ((2 * j + b) * mx + 2 * i + a).ravel()  # noqa: E731
        lower = [at(0, 0), at(2, 0), at(2, 2), at(1, 0), at(2, 1), at(1, 1)]
        upper = [at(0, 0), at(2, 2), at(0, 2), at(1, 1), at(1, 2), at(0, 1)]
        conn = np.stack([np.stack(lower, 1), np.stack(upper, 1)], 1).reshape(-1, 6)
        return nodes, conn.astype(np.int32)
    cx, cy, cz = cells
    nodes = _grid(cells)
    if distort:
        # a smooth bend that leaves the boundary planes where they are
        ext = np.array(cells) / max(cells)
        bump = 0.15 / max(cells) * np.sin(math.pi * nodes / ext).prod(1, keepdims=True)
        nodes = nodes + bump * np.cos(7.0 * nodes[:, [1, 2, 0]] + 3.0 * nodes[:, [2, 0, 1]])
    sx, sy, sz = 1, cx + 1, (cx + 1) * (cy + 1)
    k, j, i = np.meshgrid(np.arange(cz), np.arange(cy), np.arange(cx), indexing="ij")
    first = (i + sy * j + sz * k).ravel()
    if element == "hex8":
        corner = [0, sx, sx + sy, sy, sz, sz + sx, sz + sx + sy, sz + sy]
        return nodes, np.stack([first + c for c in corner], 1).astype(np.int32)
    tets = []
    for a, b, swapped in ((sx, sy, False), (sy, sz, False), (sz, sx, False),
                          (sx, sz, True), (sz, sy, True), (sy, sx, True)):
        last = first + sx + sy + sz
        mid = (first + a, first + a + b)
        tets.append(np.stack([first, mid[1], mid[0], last] if swapped
                             else [first, mid[0], mid[1], last], 1))
    return nodes, np.stack(tets, 1).reshape(-1, 4).astype(np.int32)


def _cells(case):
    return (case["nx"], case["ny"]) if case["element"] == "tri6" else (case["nx"], case["ny"],
                                                                       case["nz"])


def _velocity(nodes, seed, amplitude):
    """smooth seeded modes of wave numbers 1..4, zero on the clamped side"""
    rng = np.random.default_rng(seed)
    d = nodes.shape[1]
    v = np.zeros_like(nodes)
    for c in range(d):
        for _ in range(2):
            k, phase = rng.integers(1, 5, d), rng.uniform(0, 2 * math.pi, d)
            mode = np.ones(len(nodes))
            for a in range(d):
                mode = mode * np.sin(math.pi * k[a] * nodes[:, a] + phase[a])
            v[:, c] += amplitude * rng.uniform(0.5, 1.0) * mode
    return v * nodes[:, -1:] if d == 3 else v * nodes[:, :1]


def _state(case, nodes, seed):
    """initial velocity and blocked dofs of one mesh"""
    plane = nodes[:, -1] if nodes.shape[1] == 3 else nodes[:, 0]
    blocked = np.zeros(nodes.shape, dtype=np.uint8)
    blocked[np.abs(plane) < 1e-12] = 1
    amplitude = 0.02 if case["law"] != "elastic" else 0.01
    v = _velocity(nodes, seed, amplitude)
    v[blocked != 0] = 0.0
    return v, blocked


def _right_edge(nodes):
    return np.nonzero(nodes[:, 0] > nodes[:, 0].max() - 1e-9)[0]


def _lame(E, nu):
    return nu * E / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _time_step(case, cells, E=_E, nu=_NU):
    lam, mu = _lame(E, nu)
    factor = 0.7 if case["distort"] else 0.8
    return factor * _STABLE[case["element"]] / max(cells) / math.sqrt((lam + 2 * mu) / _RHO)


def _params(case, E=_E, nu=_NU):
    p = {"rho": _RHO, "E": E, "nu": nu}
    if case["law"] == "plastic":
        p.update(sigma_y=_SIGMA_Y, h=_HARDENING)
    return p


def _force(nodes, seed, k):
    """external force k of a stream: small, smooth, different every step"""
    w = 1.0 / len(nodes)
    f = np.zeros_like(nodes)
    f[:, k % nodes.shape[1]] = 0.02 * w * np.sin(2.0 + seed % 7 + k + 3.0 * nodes[:, 0])
    return f


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.float64).pin_memory()


def prepare(case, seed):
    """The initialised model with its initial state, as a program has it
    before its time loop (and, for a stream, its pinned buffers)."""
    element = case["element"]
    if case["flow"] == "batch":
        meshes, dts, velocity, blocked = [], [], [], []
        for k, (n, E, nu) in enumerate(_cubes(case, seed)):
            nodes, conn = _mesh(element, (n, n, n))
            meshes.append(akb.Mesh(3, nodes, conn, _TYPES[element]))
            v, b = _state(case, nodes, seed + 31 * k)
            velocity.append(v)
            blocked.append(b)
            dts.append(_time_step(case, (n, n, n), E, nu))
        model = akb.BatchModel(meshes)
        for n, E, nu in _cubes(case, seed):
            model.addMaterial(_LAWS[case["law"]], **_params(case, E, nu))
        model.setInstanceMaterials(np.arange(case["count"]))
        model.initFull(precision=case["precision"])
        model.setTimeSteps(dts)
        model.setNodal("blocked_dofs", np.concatenate(blocked))
        model.setNodal("velocity", np.concatenate(velocity))
        return {"case": case, "model": model, "views": {}}
    nodes, conn = _mesh(element, _cells(case), case["distort"])
    model = akb.SolidMechanicsModel(akb.Mesh(nodes.shape[1], nodes, conn, _TYPES[element]))
    model.addMaterial(_LAWS[case["law"]], **_params(case))
    if case["points"] == 6:
        model.setQuadratureRule(1)
    model.initFull(precision=case["precision"])
    model.setTimeStep(_time_step(case, _cells(case)))
    v, blocked = _state(case, nodes, seed)
    if element == "tri6":
        blocked[_right_edge(nodes), 0] = 1
        v[blocked != 0] = 0.0
    model.setNodal("blocked_dofs", blocked)
    model.setNodal("velocity", v)
    if element == "tri6":
        model.setPrescribedVelocityRamp(_right_edge(nodes), 0, _RAMP_SPEED, _RAMP_STEPS)
    state = {"case": case, "model": model, "views": {}}
    if case["flow"] == "stream":
        state["forces"] = [_pinned(nodes.shape) for _ in range(4)]
        for k, f in enumerate(state["forces"]):
            f.copy_(torch.from_numpy(_force(nodes, seed, k)))
        state["reads"] = [_pinned(nodes.shape) for _ in range(4)]
        state["force_arrays"] = [f.numpy() for f in state["forces"]]
        state["read_arrays"] = [r.numpy() for r in state["reads"]]
    return state


class _Device:
    """a nodal array of the model where it lies on the GPU; a tensor over it
    keeps this object, and with it the model that owns the memory"""

    def __init__(self, model, pointer, shape):
        self.model = model
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape,
                                         "typestr": "<f8", "strides": None, "version": 3}


def _view(state, field):
    model = state["model"]
    p = ctypes.c_void_p()
    rc = akb.lib().akb_model_nodal_device_pointer(model._h, field, ctypes.byref(p))
    if rc:
        raise RuntimeError("no device pointer of field %d" % field)
    view = state["views"].get(p.value)
    if view is None:
        shape = (model.mesh.getNbNodes(), model.dim)
        view = state["views"][p.value] = torch.as_tensor(_Device(model, p.value, shape),
                                                         device="cuda")
    return view


def run(state):
    case, model = state["case"], state["model"]
    if case["flow"] == "watch":
        for _ in range(case["steps"]):
            model.solveStep()
            u = model.getDisplacement()
        return {"displacement": u}
    if case["flow"] == "stream":
        tickets = []
        for k in range(case["steps"]):
            model.setNodalAsync("external_force", state["force_arrays"][k % 4])
            model.solveStep()
            tickets.append(model.getNodalAsync("displacement", state["read_arrays"][k % 4]))
            if k >= 3:
                model.waitNodalAsync(tickets[k - 3])
        model.synchronize()
        return {"read": state["reads"][(case["steps"] - 1) % 4],
                "velocity": _view(state, _VELOCITY), "acceleration": _view(state, _ACCELERATION)}
    model.solveStep(case["steps"])
    model.synchronize()  # the arrays may be read on other streams from here on
    return {"displacement": _view(state, _DISPLACEMENT), "velocity": _view(state, _VELOCITY),
            "acceleration": _view(state, _ACCELERATION)}


# -- what a pass cannot do without ---------------------------------------------------

def _sizes(case):
    """(elements, nodes) of a case"""
    per = _CELL_ELEMENTS[case["element"]]
    if case["flow"] == "batch":
        cells = [n for n, _, _ in _cubes(case, 0)]
        return sum(per * n ** 3 for n in cells), sum((n + 1) ** 3 for n in cells)
    c = _cells(case)
    order = 2 if case["element"] == "tri6" else 1
    return per * math.prod(c), math.prod(order * x + 1 for x in c)


def work(case):
    """Per step: the connectivity, the coordinates, the nodal state once in and
    once out, the mass and the flags; the plastic internals of every point
    once in and once out; per point the gradient, the law and the force."""
    E, N = _sizes(case)
    n, d = _NODES[case["element"]], 2 if case["element"] == "tri6" else 3
    q = {"tet4": 1, "hex8": 8, "tri6": case["points"]}[case["element"]]
    per_step = 4 * n * E + (8 * d + 6 * 8 * d + 9) * N
    if case["law"] == "plastic":
        sym = 6 if d == 3 else 3
        grad = 8 if case["precision"] == "fp64" else 4
        per_step += E * q * 2 * (8 * 2 * sym + grad * d * d + 8 + 8)
    law = {"elastic": 30, "neohookean": 150, "plastic": 150}[case["law"]]
    flops = E * q * (4 * n * d * d + law) + N * d * 12
    extra = 2 * 8 * d * N if case["flow"] == "stream" else 8 * d * N if case["flow"] == "watch" else 0
    return {"bytes": float(case["steps"] * (per_step + extra)), "flops": float(case["steps"] * flops)}


# -- the same steps in plain 64-bit tensors -------------------------------------------

def _shape_derivatives(element, points):
    """dN/ds (Q, d, n), the point weights and N (Q, n) of one element type"""
    if element == "tet4":
        ds = np.array([[-1.0, 0, 0, 1], [-1, 1, 0, 0], [-1, 0, 1, 0]])[None]
        return ds, np.array([1 / 6]), np.full((1, 4), 0.25)
    if element == "hex8":
        s = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                      [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)
        g = 1 / math.sqrt(3.0)
        pts = np.array([[x, y, z] for z in (-g, g) for y in (-g, g) for x in (-g, g)])
        f = 1 + pts[:, None, :] * s[None]
        ds = np.stack([s[:, 0] * f[..., 1] * f[..., 2], s[:, 1] * f[..., 0] * f[..., 2],
                       s[:, 2] * f[..., 0] * f[..., 1]], 1) / 8
        return ds, np.ones(8), f.prod(2) / 8
    if points == 6:
        r, t = math.sqrt(10.0), math.sqrt(38.0 - 44.0 * math.sqrt(0.4))
        a, b = (8 - r + t) / 18, (8 - r - t) / 18
        q = math.sqrt(213125.0 - 53320.0 * r)
        pts = np.array([[b, b], [1 - 2 * b, b], [b, 1 - 2 * b], [a, 1 - 2 * a], [a, a], [1 - 2 * a, a]])
        w = np.array([(620 - q) / 7440] * 3 + [(620 + q) / 7440] * 3)
    else:
        pts = np.array([[1 / 6, 1 / 6], [2 / 3, 1 / 6], [1 / 6, 2 / 3]])
        w = np.full(3, 1 / 6)
    x, y = pts[:, 0], pts[:, 1]
    z, o = 1 - x - y, np.zeros(len(pts))
    N = np.stack([z * (2 * z - 1), x * (2 * x - 1), y * (2 * y - 1), 4 * z * x, 4 * x * y, 4 * y * z], 1)
    dx = np.stack([1 - 4 * z, 4 * x - 1, o, 4 * (z - x), 4 * y, -4 * y], 1)
    dy = np.stack([1 - 4 * z, o, 4 * y - 1, -4 * x, 4 * x, 4 * (z - y)], 1)
    return np.stack([dx, dy], 1), w, N


def _elastic(g, lam, mu):
    d = g.shape[-1]
    tr = g.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
    eye = torch.eye(d, dtype=g.dtype, device=g.device)
    return lam * tr * eye + mu * (g + g.transpose(-1, -2))


def _neohookean(g, lam, mu):
    """first Piola-Kirchhoff stress, P[i, j] = mu F + (lambda ln J - mu) F^-T"""
    F = g + torch.eye(3, dtype=g.dtype, device=g.device)
    r = F.unbind(-2)
    cof = torch.stack([torch.linalg.cross(r[1], r[2]), torch.linalg.cross(r[2], r[0]),
                       torch.linalg.cross(r[0], r[1])], -2)
    J = (r[0] * cof[..., 0, :]).sum(-1)[..., None, None]
    return mu * F + (lam * torch.log(J) - mu) / J * cof


class _Plastic:
    """radial return with linear isotropic hardening, small strains, plane"""

    def __init__(self):
        self.g = self.s = self.iso = None

    def __call__(self, g, lam, mu):
        if self.g is None:
            self.g, self.s = torch.zeros_like(g), torch.zeros_like(g)
            self.iso = torch.zeros(g.shape[:-2], dtype=g.dtype, device=g.device)
        dg = g - self.g
        trial = self.s + _elastic(dg, lam, mu)
        third = trial.diagonal(dim1=-2, dim2=-1).sum(-1) / 3
        dev = trial - third[..., None, None] * torch.eye(2, dtype=g.dtype, device=g.device)
        eff = torch.sqrt(1.5 * ((dev * dev).sum((-1, -2)) + third * third))
        flow = eff - self.iso - _SIGMA_Y
        dp = torch.where(flow > 0, flow / (3 * mu + _HARDENING), torch.zeros_like(flow))
        deps = dev * (1.5 * dp / torch.where(eff > 0, eff, torch.ones_like(eff)))[..., None, None]
        self.s = self.s + _elastic(dg - deps, lam, mu)
        self.iso = self.iso + _HARDENING * dp
        self.g = g
        return self.s


def _advance(case, nodes, conn, seed, lam, mu, dt, velocity, blocked, reads=False):
    """`steps` central-difference steps of one mesh; lam and mu are numbers or
    one value per element, dt a number or one value per node"""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f8 = dict(dtype=torch.float64, device=dev)
    X = torch.as_tensor(nodes, **f8)
    c = torch.as_tensor(conn, device=dev).long()
    E, n = c.shape
    N, d = X.shape
    ds, w, shape = _shape_derivatives(case["element"], case["points"])
    Q = len(w)
    B = torch.empty(E, n, Q * d, **f8)       # dN_a/dx_j of point q at [e, a, q d + j]
    wJ = torch.empty(E, Q, **f8)
    for q in range(Q):
        D = torch.as_tensor(ds[q], **f8)
        J = D @ X[c]                          # dX_j/ds_k at [e, k, j]
        B[:, :, q * d:(q + 1) * d] = torch.linalg.solve(J, D.expand(E, d, n)).transpose(1, 2)
        wJ[:, q] = torch.linalg.det(J) * w[q]
    per = torch.zeros(E, n, **f8)
    if case["element"] == "tri6":
        per += wJ.sum(1, keepdim=True) * torch.tensor([1 / 12] * 3 + [1 / 4] * 3, **f8)
    else:
        per += wJ @ torch.as_tensor(shape, **f8)
    mass = torch.zeros(N, **f8).index_add_(0, c.reshape(-1), _RHO * per.reshape(-1))[:, None]
    law = {"elastic": _elastic, "neohookean": _neohookean, "plastic": _Plastic()}[case["law"]]
    free = torch.as_tensor(blocked == 0, device=dev).double()
    v = torch.as_tensor(velocity, **f8).clone()
    u, a = torch.zeros_like(v), torch.zeros_like(v)
    edge = torch.as_tensor(_right_edge(nodes), device=dev) if case["element"] == "tri6" else None
    pulled = 0.0
    for k in range(case["steps"]):
        u = u + free * (dt * v + 0.5 * dt * dt * a)
        if edge is not None:
            pulled += dt * _RAMP_SPEED * min(1.0, (k + 1) / _RAMP_STEPS)
            u[edge, 0] = pulled
        f = torch.zeros_like(u)
        for lo in range(0, E, 1 << 19):
            hi = E if case["law"] == "plastic" else min(E, lo + (1 << 19))
            g = torch.bmm(u[c[lo:hi]].transpose(1, 2), B[lo:hi])      # [e, i, q d + j]
            g = g.reshape(-1, d, Q, d).transpose(1, 2)                # [e, q, i, j]
            l, m = (x[lo:hi] if isinstance(x, torch.Tensor) else x for x in (lam, mu))
            P = law(g, l, m) * wJ[lo:hi, :, None, None]
            r = torch.bmm(B[lo:hi], P.transpose(2, 3).reshape(hi - lo, Q * d, d))
            f.index_add_(0, c[lo:hi].reshape(-1), -r.reshape(-1, d))
            if hi == E:
                break
        if case["flow"] == "stream":
            f += torch.as_tensor(_force(nodes, seed, k % 4), **f8)
        new = free * (f / mass)
        v = v + free * (0.5 * dt * (a + new))
        a = new
    return u, v, a


def exact(case, seed):
    element = case["element"]
    if case["flow"] == "batch":
        X, C, V, K, dts, lams, mus, off = [], [], [], [], [], [], [], 0
        for k, (n, E, nu) in enumerate(_cubes(case, seed)):
            nodes, conn = _mesh(element, (n, n, n))
            v, b = _state(case, nodes, seed + 31 * k)
            lam, mu = _lame(E, nu)
            X.append(nodes), C.append(conn.astype(np.int64) + off), V.append(v), K.append(b)
            dts.append(np.full(len(nodes), _time_step(case, (n, n, n), E, nu)))
            lams.append(np.full(len(conn), lam)), mus.append(np.full(len(conn), mu))
            off += len(nodes)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        wide = lambda x, *s: torch.as_tensor(np.concatenate(x), device=dev).reshape(*s)  # noqa: E731
        u, v, a = _advance(case, np.concatenate(X), np.concatenate(C), seed,
                           wide(lams, -1, 1, 1, 1), wide(mus, -1, 1, 1, 1), wide(dts, -1, 1),
                           np.concatenate(V), np.concatenate(K))
        return {"displacement": u, "velocity": v, "acceleration": a}
    nodes, conn = _mesh(element, _cells(case), case["distort"])
    v, blocked = _state(case, nodes, seed)
    if element == "tri6":
        blocked[_right_edge(nodes), 0] = 1
        v[blocked != 0] = 0.0
    lam, mu = _lame(_E, _NU)
    u, v, a = _advance(case, nodes, conn, seed, lam, mu, _time_step(case, _cells(case)), v, blocked)
    if case["flow"] == "watch":
        return {"displacement": u}
    if case["flow"] == "stream":
        return {"read": u, "velocity": v, "acceleration": a}
    return {"displacement": u, "velocity": v, "acceleration": a}
