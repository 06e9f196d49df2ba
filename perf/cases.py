"""The calls by which this library's speed is judged: exterior Burton-Miller
solves, new designs and pressure maps, through the public Python interface
(CudaBemSolver), over the range of meshes and requests it serves.

A case names a task, a mesh family and size, a solver form and a request:

* task "sweep": the mesh's solver and its interaction plan are kept, as a
  frequency sweep keeps them; one pass solves every frequency of the raster.
* task "design": one pass takes a mesh that was not seen before through
  validation, planning and solving, as an optimiser or a serving loop does.
* task "samples": one pass maps the pressure of a solved frequency at points
  around the source.

Meshes: "octahedral" and "icosphere" (size: refinements; a slightly ellipsoidal
cabinet of 0.1 m), "rings" (ring-meshed sphere, size: edge length in mm) and
"horn" (exponential horn shell, size: edge length in mm; wall in mm). The seed
moves the axes, the driver velocities and the observers; triangles and frequencies
belong to the case.
"""
import math

import numpy as np
import torch

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

SOUND_SPEED, DENSITY = 343.0, 1.21


def _case(name, task, mesh, size, low, high, frequencies, **more):
    case = {"name": name, "task": task, "mesh": mesh, "size": size, "low": low, "high": high,
            "frequencies": frequencies, "precision": "fp64", "acceleration": "dense", "drivers": 1, "observers": 3,
            "far": False, "wall": 3.0}
    case.update(more)
    return case


def listed():
    return [
        # one frequency on a small closed cabinet: an interactive edit, or one point of an
        # optimiser's line search; latency and launches count
        _case("point 512 triangles", "sweep", "octahedral", 3, 1000.0, 1000.0, 1),
        # the headline sweep, in both forms: 32 log frequencies of a 0.1 m source
        _case("sweep 1280 mixed", "sweep", "icosphere", 3, 100.0, 5000.0, 32, precision="mixed"),
        _case("sweep 1280 fp64", "sweep", "icosphere", 3, 100.0, 5000.0, 32),
        # a two-driver cabinet: both drivers solved at once, an ordinary mesh
        _case("two drivers 5120 fp64", "sweep", "icosphere", 4, 500.0, 4000.0, 2, drivers=2),
        # a directivity balloon: 5 degree grid of far-field directions, two drivers
        _case("balloon 1280 fp64", "sweep", "icosphere", 3, 250.0, 4000.0, 8, drivers=2, observers=2664, far=True),
        # horns, the library's subject: a throat driver, odd triangle counts, facing skins across
        # the wall; the first at a medium mesh, the next two at the full 8 kHz mesh
        _case("horn 8k mixed", "sweep", "horn", 9.0, 250.0, 2500.0, 3, precision="mixed"),
        _case("horn 12.8k fp64", "sweep", "horn", 7.14583333333, 2000.0, 2000.0, 1),
        _case("horn 12.8k mixed", "sweep", "horn", 7.14583333333, 2000.0, 2000.0, 1, precision="mixed"),
        # the fast-multipole forms, for meshes where the dense matrix is too large a price
        _case("horn 8k multipole fp64", "sweep", "horn", 9.0, 2000.0, 2000.0, 1, acceleration="fast_multipole"),
        _case("horn 8k multipole mixed", "sweep", "horn", 9.0, 1500.0, 1500.0, 1, acceleration="fast_multipole",
              precision="mixed"),
        # a horn the session has not seen: validation, planning and four frequencies
        _case("new horn 3.6k mixed", "design", "horn", 14.8, 400.0, 3200.0, 4, precision="mixed", wall=18.0),
        # a pressure map in front of the source, from near the surface to 1 m
        _case("map 4096 points", "samples", "icosphere", 3, 2000.0, 2000.0, 1, observers=4096),
    ]


# Triangle counts of a mesh by its size, within a few percent, for draw() and work().
def _triangles(case):
    if case["mesh"] == "octahedral":
        return 8 * 4 ** case["size"]
    if case["mesh"] == "icosphere":
        return 20 * 4 ** case["size"]
    if case["mesh"] == "rings":
        return 2.56e5 / case["size"] ** 2
    return 12756 * (7.14583333333 / case["size"]) ** 2


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    task = rng.choice(("sweep", "sweep", "sweep", "sweep", "sweep", "design", "samples"))
    multipole = task == "sweep" and rng.random() < 0.2
    mesh = "horn" if multipole and rng.random() < 0.5 else rng.choice(("rings", "rings", "horn"))
    if task == "samples":
        mesh = "rings"
    low_t, high_t = (4000, 8000) if multipole else (300, 4000) if task == "design" else (300, 9000)
    if mesh == "horn":
        low_t = max(low_t, 2500)  # coarser edges do not follow the throat
    if task == "samples":
        high_t = 3000
    triangles = _log(rng, low_t, high_t)
    case = _case("", task, mesh, 1.0, 0.0, 0.0, 1)
    if mesh == "rings":
        case["size"] = round(math.sqrt(2.56e5 / triangles), 3)
        longest = 1.75e-3 * case["size"]
    else:
        case["size"] = round(7.14583333333 * math.sqrt(12756 / triangles), 3)
        longest = 1.75e-3 * case["size"]
        case["wall"] = round(max(3.0, 1.2 * case["size"]), 3)
    top = min(12000.0, 1.8 / longest * SOUND_SPEED / (2 * math.pi))
    if multipole:
        case["acceleration"], top = "fast_multipole", min(top, 2500.0)
    case["high"] = round(_log(rng, 0.25 * top, top), 2)
    case["low"] = round(_log(rng, 100.0, case["high"]), 2)
    if task == "samples":
        case["low"], case["observers"] = case["high"], int(_log(rng, 16, 4096))
    elif not multipole:
        most = max(1.0, min(32.0, 1.4e8 / triangles ** 2))
        case["frequencies"] = int(_log(rng, 1, most + 0.999))
        case["far"] = rng.random() < 0.3
        case["observers"] = int(_log(rng, 1, 2664 if case["far"] else 64))
        case["drivers"] = rng.choice((1, 1, 2, 3)) if mesh == "rings" else 1
    if case["frequencies"] == 1:
        case["low"] = case["high"]
    if task != "samples":
        case["precision"] = rng.choice(("fp64", "mixed"))
    del case["name"]
    return case


# -- inputs ------------------------------------------------------------------


def _mesh(case, axes):
    size = case["size"]
    if case["mesh"] == "horn":
        wall = 1e-3 * case["wall"]
        base = meshes.exponential_horn(h=1e-3 * size, wall=wall, rear=wall)
        return meshes.SurfaceMesh(base.vertices * axes, base.triangles, base.face_ids, base.boundary)
    if case["mesh"] == "rings":
        base = meshes.revolved_sphere(h=1e-3 * size)
    else:
        base = (meshes.octahedral_sphere if case["mesh"] == "octahedral" else meshes.icosphere)(size)
    faces = np.ones(base.triangle_count, np.uint32)
    driven = np.full(base.triangle_count, meshes.DRIVEN, np.uint8)
    drivers = case["drivers"]
    if drivers > 1:  # caps around the vertical axis, and a rigid body between them
        z = base.vertices[base.triangles].mean(1)[:, 2] / 0.1
        band = np.minimum(((z + 1.0) / 2.0 * (2 * drivers - 1)).astype(int), 2 * drivers - 2)
        faces = np.where(band % 2 == 0, band // 2 + 1, drivers + 1)
        driven = np.where(band % 2 == 0, meshes.DRIVEN, meshes.WALL)
    return meshes.SurfaceMesh(base.vertices * axes, base.triangles, faces, driven)


def _inputs(case, seed):
    """Mesh, frequencies, driver velocities (one excitation per driver), observers."""
    rng = np.random.default_rng([seed, 17])
    axes = rng.uniform(0.96, 1.04, 3)
    mesh = _mesh(case, axes)
    n = case["frequencies"]
    frequencies = [float(f) for f in np.round(np.geomspace(case["low"], case["high"], n) if n > 1 else [case["high"]], 3)]
    velocities = rng.uniform(0.2, 1.0, case["drivers"]) * np.exp(1j * rng.uniform(-math.pi, math.pi, case["drivers"]))
    extent = float(np.linalg.norm(mesh.vertices, axis=1).max())
    direction = rng.normal(size=(case["observers"], 3))
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    if case["task"] == "samples":  # from 3 mm off the surface, denser towards it, and some points inside the body
        gap = np.exp(rng.uniform(math.log(0.03), math.log(9.0), case["observers"]))
        radius = np.where(rng.random(case["observers"]) < 0.05, 0.07, 0.1 * (1 + gap))
        direction = direction * axes
    else:
        radius = extent * rng.uniform(1.3, 10.0, case["observers"])
    return mesh, frequencies, velocities, direction * radius[:, None]


def _request(case, frequencies, velocities, observers, raster):
    return hs.BemRequest(
        frequencies=frequencies,
        excitations=[hs.BemExcitation("driver %d" % d, [hs.FaceVelocity(d + 1, complex(v))])
                     for d, v in enumerate(velocities)],
        observers=observers, medium=hs.AcousticMedium(DENSITY, SOUND_SPEED),
        numerics=hs.BemNumerics(precision=case["precision"], acceleration=case["acceleration"]),
        far_field=hs.FarFieldObservation() if case["far"] else None, interaction_plan_frequencies=raster)


def _monopoles(seed):
    rng = np.random.default_rng([seed, 29])
    return rng.uniform(-0.03, 0.03, (3, 3)), rng.normal(size=3) + 1j * rng.normal(size=3)


def _radiated(mesh, frequency, seed):
    """Traces of a field radiated by monopoles inside the body: pressure per vertex and its
    normal derivative per triangle, as a solve leaves them."""
    k = 2 * math.pi * frequency / SOUND_SPEED
    where, strength = _monopoles(seed)
    corner = mesh.vertices[mesh.triangles]
    normal = np.cross(corner[:, 1] - corner[:, 0], corner[:, 2] - corner[:, 0])
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    trace, slope = 0, 0
    for x, s in zip(where, strength):
        d = mesh.vertices - x
        r = np.linalg.norm(d, axis=1)
        trace = trace + s * np.exp(-1j * k * r) / (4 * math.pi * r)
        d = corner.mean(1) - x
        r = np.linalg.norm(d, axis=1)
        slope = slope - s * np.exp(-1j * k * r) / (4 * math.pi * r) * (1j * k + 1 / r) * (d * normal).sum(1) / r
    return trace, slope


def prepare(case, seed):
    mesh, frequencies, velocities, observers = _inputs(case, seed)
    state = {"case": case, "mesh": mesh}
    if case["task"] == "samples":
        trace, slope = _radiated(mesh, frequencies[0], seed)
        surface = trace[mesh.triangles].mean(1)
        state.update(solver=hs.CudaBemSolver(mesh), points=observers, frequency=frequencies[0],
                     solution=hs.BemExcitationResult("driver 0", np.zeros(0), [], 0, 0.0, 0, 0, 0.0,
                                                     hs.BemBoundaryData(surface, trace, slope)))
        return state
    state["request"] = _request(case, frequencies, velocities, observers, frequencies)
    if case["task"] == "sweep":
        # the solver keeps the mesh and its interaction plan: made by its first solve, of one frequency
        state["solver"] = hs.CudaBemSolver(mesh)
        state["solver"].solve(_request(case, frequencies[:1], velocities, observers, frequencies))
    return state


def _whole(result):
    """The solved fields: one array [frequency, excitation, ...] of each kind."""
    rows = [[e for e in f.excitations] for f in result.frequencies]

    def stack(value):
        return np.array([[value(e) for e in row] for row in rows])

    return {"trace": stack(lambda e: e.boundary.pressure_trace), "surface": stack(lambda e: e.boundary.surface_pressure),
            "derivative": stack(lambda e: e.boundary.normal_derivative), "observers": stack(lambda e: e.observer_pressure),
            "impedance": stack(lambda e: [[i.mean_pressure, i.volume_velocity, i.volume_impedance] for i in e.impedances])}


def run(state):
    task = state["case"]["task"]
    if task == "samples":
        samples = state["solver"].pressure_field(state["frequency"], state["solution"], state["points"],
                                                 medium=hs.AcousticMedium(DENSITY, SOUND_SPEED))
        return {"pressure": np.array([s.pressure for s in samples]),
                "status": np.array([int(s.status) for s in samples], np.int32)}
    if task == "design":
        with hs.CudaBemSolver(state["mesh"]) as solver:
            return _whole(solver.solve(state["request"]))
    return _whole(state["solver"].solve(state["request"]))


# -- what a pass cannot do without -------------------------------------------


def work(case):
    t = float(_triangles(case))
    n, f, e, o = t / 2, float(case["frequencies"]), float(case["drivers"]), float(case["observers"])
    inputs = t * (3 * 4 + 5) + n * 24 + o * 24
    outputs = f * e * (n + 2 * t + o) * 16
    if case["task"] == "samples":  # 12 samples of about 40 operations for each point and triangle
        return {"bytes": t * 16 + n * 16 + inputs + o * 20, "flops": o * t * 12 * 40}
    field = f * e * o * t * 6 * 40
    if case["acceleration"] == "fast_multipole":
        # near entries of about 500 neighbours a vertex by 36-point panel pairs, and twenty
        # applications of the operator; its expansions at about 10 degrees, six channels
        near = n * 500
        return {"bytes": f * 20 * near * 20 + inputs + outputs,
                "flops": f * (near * 12 * 36 * 85 + 20 * e * (8 * near + 6 * n / 8 * 189 * 1000 * 8)) + field}
    # every unordered pair of triangles once by 36 samples of 85 operations, the matrix
    # written, factored and read, and the fields
    return {"bytes": f * n * n * 16 * 3 + inputs + outputs,
            "flops": f * (t * t / 2 * 36 * 85 + 8 / 3 * n ** 3 + 16 * e * n * n) + field}


# -- the same integrals in 64 bits, by plain torch -----------------------------


def _tensor_rule(n, splits=0):
    """Gauss-Legendre points collapsed onto the unit triangle, on 4**splits equal
    parts of it: barycentric coordinates (Q, 3) and weights of total one half."""
    g, w = np.polynomial.legendre.leggauss(n)
    g, w = (g + 1) / 2, w / 2
    u, v = np.meshgrid(g, g, indexing="ij")
    points = np.stack([u * (1 - v), u * v], -1).reshape(-1, 2)
    weights = (np.outer(w, w) * u).reshape(-1)
    for _ in range(splits):
        h = points / 2
        points = np.concatenate([h, h + [0.5, 0], h + [0, 0.5], [0.5, 0.5] - h])
        weights = np.concatenate([weights / 4] * 4)
    return np.concatenate([1 - points.sum(1, keepdims=True), points], 1), weights


def _touching_rule(shared, n):
    """Sauter and Schwab's regularising coordinates for two triangles with `shared` common
    vertices (the first ones of both): barycentrics of both (Q, 3) and weights."""
    g, w = np.polynomial.legendre.leggauss(n)
    g, w = (g + 1) / 2, w / 2
    xi, a, b, c = (x.reshape(-1) for x in np.meshgrid(g, g, g, g, indexing="ij"))
    weight = (w[:, None, None, None] * w[:, None, None] * w[:, None] * w).reshape(-1)
    one = np.ones_like(xi)
    if shared == 3:
        first = [((one, 1 - a + a * b), (1 - a * b * c, 1 - a)), ((one, a * (1 - b + b * c)), (1 - a * b, a * (1 - b))),
                 ((one, a * (1 - b)), (1 - a * b * c, a * (1 - b * c)))]
        sectors = [(x, y, a * a * b) for x, y in first] + [(y, x, a * a * b) for x, y in first]
    elif shared == 2:
        sectors = [((one, a * c), (1 - a * b, a * (1 - b)), a * a),
                   ((one, a), (1 - a * b * c, a * b * (1 - c)), a * a * b),
                   ((1 - a * b, a * (1 - b)), (one, a * b * c), a * a * b),
                   ((1 - a * b * c, a * b * (1 - c)), (one, a), a * a * b),
                   ((1 - a * b * c, a * (1 - b * c)), (one, a * b), a * a * b)]
    else:
        sectors = [((one, a), (b, b * c), b), ((b, b * c), (one, a), b)]

    def corners(p):  # (p1, p2) with 0 <= p2 <= p1 <= 1: the first vertex at the origin
        return np.stack([1 - xi * p[0], xi * (p[0] - p[1]), xi * p[1]], 1)

    return (np.concatenate([corners(x) for x, _, _ in sectors]), np.concatenate([corners(y) for _, y, _ in sectors]),
            np.concatenate([weight * xi ** 3 * j for _, _, j in sectors]))


class _Boundary:
    """Galerkin P1 / DP0 Burton-Miller system of a closed mesh, rules well above the accuracy asked for."""

    def __init__(self, mesh):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        self.tri = torch.as_tensor(mesh.triangles.astype(np.int64), device=self.device)
        self.n, self.t = mesh.vertex_count, mesh.triangle_count
        p = self.corner = self.tensor(mesh.vertices)[self.tri]
        cross = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        self.area = torch.linalg.norm(cross, dim=1) / 2
        self.normal = cross / (2 * self.area[:, None])
        opposite = torch.stack([p[:, 2] - p[:, 1], p[:, 0] - p[:, 2], p[:, 1] - p[:, 0]], 1)
        self.curl = opposite / (2 * self.area[:, None, None])
        triangles = mesh.triangles.astype(np.int64)
        common = [set() for _ in range(self.t)]
        at = [[] for _ in range(self.n)]
        for t, nodes in enumerate(triangles):
            for v in nodes:
                at[v].append(t)
        for t, nodes in enumerate(triangles):
            common[t] = {s for v in nodes for s in at[v]}
        self.touching = {1: [], 2: [], 3: []}
        for t in range(self.t):
            for s in common[t]:
                shared = [v for v in triangles[t] if v in triangles[s]]
                order = [[list(x).index(v) for v in shared] for x in (triangles[t], triangles[s])]
                order = [o + [i for i in range(3) if i not in o] for o in order]
                self.touching[len(shared)].append((t, s, *order[0], *order[1]))
        centre = p.mean(1)
        edge = torch.linalg.norm(opposite, dim=2).amax(1)
        close = torch.cdist(centre, centre) < 1.1 * (edge[:, None] + edge[None])
        for pairs in self.touching.values():
            if pairs:
                q = torch.tensor(pairs, device=self.device)
                close[q[:, 0], q[:, 1]] = False
        self.near = close.nonzero()
        self.apart = ~close
        for pairs in self.touching.values():
            if pairs:
                q = torch.tensor(pairs, device=self.device)
                self.apart[q[:, 0], q[:, 1]] = False

    def tensor(self, x):
        return torch.as_tensor(np.asarray(x), dtype=torch.float64, device=self.device)

    def _kernels(self, d, normal_x, normal_y, k):
        """Green's function at y - x = d, and its derivatives along both normals."""
        r2 = (d * d).sum(-1)
        r = r2.sqrt()
        green = torch.polar(1 / (4 * math.pi * r), -k * r)
        slope = green * torch.complex(torch.ones_like(r), k * r) / r2
        return green, -slope * (d * normal_y).sum(-1), slope * (d * normal_x).sum(-1)

    def _add(self, rows, cols, test, trial, g, gy, gx, k):
        """Adds pair blocks (P, 3, 3), (P, 3, 3), (P, 3) at nodes rows and cols (P, 3)."""
        alpha = -1j / k
        cc = torch.einsum("pix,pjx->pij", *(torch.gather(self.curl[t], 1, o[..., None].expand(-1, -1, 3))
                                            for t, o in ((test, rows[1]), (trial, cols[1]))))
        nn = (self.normal[test] * self.normal[trial]).sum(1)[:, None, None]
        block = -gy + alpha * (g.sum((1, 2))[:, None, None] * cc - k * k * nn * g)
        at = (rows[0][:, :, None] * self.n + cols[0][:, None, :]).reshape(-1)
        torch.view_as_real(self.matrix).view(-1, 2).index_add_(0, at, torch.view_as_real(block.reshape(-1)))
        at = (rows[0] * self.t + trial[:, None]).reshape(-1)
        side = -g.sum(2) - alpha * gx
        torch.view_as_real(self.side).view(-1, 2).index_add_(0, at, torch.view_as_real(side.reshape(-1)))

    def _pairs(self, test, trial, order_x, order_y, bx, by, w, k):
        """Pairs by one rule of both triangles' points together, (Q, 3), (Q, 3), (Q)."""
        step = max(1, int(4e6 // len(w)))
        bx, by, w = self.tensor(bx), self.tensor(by), self.tensor(w).to(torch.complex128)
        for i in range(0, len(test), step):
            a, b, ox, oy = test[i:i + step], trial[i:i + step], order_x[i:i + step], order_y[i:i + step]
            px = torch.gather(self.corner[a], 1, ox[..., None].expand(-1, -1, 3))
            py = torch.gather(self.corner[b], 1, oy[..., None].expand(-1, -1, 3))
            d = torch.einsum("qi,pix->pqx", by, py) - torch.einsum("qi,pix->pqx", bx, px)
            g, gy, gx = self._kernels(d, self.normal[a][:, None], self.normal[b][:, None], k)
            scale = (4 * self.area[a] * self.area[b])[:, None] * w
            both = (bx[:, :, None] * by[:, None, :]).reshape(len(w), 9).to(torch.complex128)
            blocks = [((v * scale) @ both).view(-1, 3, 3) for v in (g, gy)]
            self._add((torch.gather(self.tri[a], 1, ox), ox), (torch.gather(self.tri[b], 1, oy), oy), a, b, *blocks,
                      (gx * scale) @ bx.to(torch.complex128), k)

    def _far(self, k, n=4):
        rule, w = _tensor_rule(n)
        q = len(w)
        rule, w = self.tensor(rule), self.tensor(w)
        points = torch.einsum("qi,tix->tqx", rule, self.corner)
        basis = (rule * w[:, None]).to(torch.complex128)
        alone = torch.arange(3, device=self.device)
        step = max(1, int(4e6 // (q * q * self.t)))
        for i in range(0, self.t, step):
            a = torch.arange(i, min(i + step, self.t), device=self.device)
            test, trial = (x.reshape(-1) for x in torch.meshgrid(a, torch.arange(self.t, device=self.device), indexing="ij"))
            keep = self.apart[test, trial]
            test, trial = test[keep], trial[keep]
            d = points[trial][:, None] - points[test][:, :, None]
            g, gy, gx = self._kernels(d, self.normal[test][:, None, None], self.normal[trial][:, None, None], k)
            scale = (4 * self.area[test] * self.area[trial])[:, None, None]
            blocks = [torch.einsum("qi,pqj->pij", basis, v @ basis) * scale for v in (g, gy)]
            gx = (gx @ w.to(torch.complex128)) @ basis * scale[:, 0]
            order = alone.expand(len(test), 3)
            self._add((self.tri[test], order), (self.tri[trial], order), test, trial, *blocks, gx, k)

    def solve(self, k, slopes):
        """P1 pressures (E, N) for normal derivatives (E, T)."""
        self.matrix = torch.zeros(self.n, self.n, dtype=torch.complex128, device=self.device)
        self.side = torch.zeros(self.n, self.t, dtype=torch.complex128, device=self.device)
        alone = torch.arange(3, device=self.device)
        self._far(k)
        rule, w = _tensor_rule(4, 1)
        bx, by = (x.reshape(-1, 3) for x in (np.repeat(rule, len(rule), 0), np.tile(rule, (len(rule), 1))))
        order = alone.expand(len(self.near), 3)
        self._pairs(self.near[:, 0], self.near[:, 1], order, order, bx, by, np.outer(w, w).reshape(-1), k)
        for shared, pairs in self.touching.items():
            if pairs:
                p = torch.tensor(pairs, device=self.device)
                self._pairs(p[:, 0], p[:, 1], p[:, 2:5], p[:, 5:8], *_touching_rule(shared, 7), k)
        mass = (torch.eye(3, device=self.device, dtype=torch.float64) + 1) / 12
        at = (self.tri[:, :, None] * self.n + self.tri[:, None, :]).reshape(-1)
        half = torch.zeros(self.n * self.n, dtype=torch.float64, device=self.device)
        half.index_add_(0, at, (self.area[:, None, None] * mass / 2).reshape(-1))
        flux = torch.zeros(self.n * self.t, dtype=torch.float64, device=self.device)
        at = (self.tri * self.t + torch.arange(self.t, device=self.device)[:, None]).reshape(-1)
        flux.index_add_(0, at, (self.area / 6)[:, None].expand(-1, 3).reshape(-1))
        a = self.matrix + half.view(self.n, self.n)
        b = self.side + 1j / k * flux.view(self.n, self.t)
        return torch.linalg.solve(a, b @ slopes.T).T

    def field(self, k, trace, slope, points, splits, far=None):
        """Pressure (E, O) at points, or at far-field directions for the reference distance `far`."""
        rule, w = _tensor_rule(4, splits)
        rule, w = self.tensor(rule), self.tensor(w)
        y = torch.einsum("qi,tix->tqx", rule, self.corner).reshape(-1, 3)
        weight = (2 * self.area[:, None] * w).reshape(-1).to(torch.complex128)
        normal = self.normal.repeat_interleave(len(w), 0)
        p = torch.einsum("qi,eti->etq", rule.to(torch.complex128), trace[:, self.tri]).flatten(1) * weight
        s = slope.repeat_interleave(len(w), 1) * weight
        out = []
        step = max(1, int(2e7 // len(y)))
        for i in range(0, len(points), step):
            x = points[i:i + step]
            if far is not None:
                green = torch.polar(torch.full((len(x), len(y)), 1 / (4 * math.pi * far), device=self.device,
                                               dtype=torch.float64), k * (x @ y.T - far))
                out.append((p @ (green * 1j * k * (x @ normal.T)).T) - s @ green.T)
                continue
            d = y[None] - x[:, None]
            green, gy, _ = self._kernels(d, normal, normal, k)
            out.append(p @ gy.T - s @ green.T)
        return torch.cat(out, 1)


def _exact_samples(case, seed):
    mesh, frequencies, _, points = _inputs(case, seed)
    trace, slope = _radiated(mesh, frequencies[0], seed)
    b = _Boundary(mesh)
    k = 2 * math.pi * frequencies[0] / SOUND_SPEED
    trace, slope = (torch.as_tensor(x, device=b.device)[None] for x in (trace, slope))
    x = b.tensor(points)
    p = b.field(k, trace, slope, x, 1)[0]
    # panels close to a point: by parts as small as the distance asks for
    centre, edge = b.corner.mean(1), torch.linalg.norm(b.corner - b.corner.roll(1, 1), dim=2).amax()
    distance = torch.cdist(x, centre)
    for splits, low, high in ((3, 0.8, 2.5), (5, 0.0, 0.8)):
        at, panel = ((distance >= low * edge) & (distance < high * edge)).nonzero().T
        for s, sign in ((1, -1), (splits, 1)):
            rule, w = (b.tensor(v) for v in _tensor_rule(4, s))
            for i in range(0, len(at), 400):
                o, t = at[i:i + 400], panel[i:i + 400]
                d = torch.einsum("qi,pix->pqx", rule, b.corner[t]) - x[o][:, None]
                green, gy, _ = b._kernels(d, b.normal[t][:, None], b.normal[t][:, None], k)
                values = trace[0, b.tri[t]] @ rule.T.to(torch.complex128)
                panels = ((values * gy - slope[0, t][:, None] * green) * (2 * b.area[t][:, None] * w)).sum(1)
                torch.view_as_real(p).index_add_(0, o, sign * torch.view_as_real(panels))
    # the solid angle of the surface tells inside from outside; a point within the
    # exclusion distance has no pressure either
    a, c, d = (b.corner[None, :, i] - x[:, None] for i in range(3))
    la, lc, ld = (torch.linalg.norm(v, dim=2) for v in (a, c, d))
    num = (a * torch.linalg.cross(c, d)).sum(2)
    den = la * lc * ld + (a * c).sum(2) * ld + (c * d).sum(2) * la + (d * a).sum(2) * lc
    inside = (2 * torch.atan2(num, den)).sum(1).abs() > 2 * math.pi
    p[inside] = 0
    return {"pressure": p.cpu().numpy(), "status": None}


def exact(case, seed):
    if case["task"] == "samples":
        return _exact_samples(case, seed) if _triangles(case) * case["observers"] < 6e6 else None
    mesh, frequencies, velocities, observers = _inputs(case, seed)
    drivers = case["drivers"]
    panel = np.zeros((drivers, mesh.triangle_count), complex)
    for d in range(drivers):
        panel[d, mesh.face_ids == d + 1] = velocities[d]
    slopes = np.array([-1j * DENSITY * 2 * math.pi * f * panel for f in frequencies])
    out = {"trace": None, "surface": None, "derivative": slopes, "observers": None, "impedance": None}
    # a wall of a few millimetres, or many triangles, takes too many samples for this
    if case["mesh"] == "horn" or case["frequencies"] * mesh.triangle_count ** 2 > 6e7 or mesh.triangle_count > 3000:
        return out
    b = _Boundary(mesh)
    x = b.tensor(observers)
    if case["far"]:
        x = x / torch.linalg.norm(x, dim=1, keepdim=True)
    traces, fields = [], []
    for f, s in zip(frequencies, slopes):
        k = 2 * math.pi * f / SOUND_SPEED
        s = torch.as_tensor(s, device=b.device)
        trace = b.solve(k, s)
        traces.append(trace)
        fields.append(b.field(k, trace, s, x, 1, 1.0 if case["far"] else None))
    trace = torch.stack(traces).cpu().numpy()
    surface = trace[:, :, mesh.triangles].mean(3)
    area = b.area.cpu().numpy()
    face = [mesh.face_ids == d + 1 for d in range(drivers)]
    mean = np.stack([surface[:, d][:, face[d]] @ area[face[d]] / area[face[d]].sum() for d in range(drivers)], 1)
    volume = np.broadcast_to([velocities[d] * area[face[d]].sum() for d in range(drivers)], mean.shape)
    out.update(trace=trace, surface=surface, observers=torch.stack(fields).cpu().numpy(),
               impedance=np.stack([mean, volume, mean / volume], 2)[:, :, None])
    return out
