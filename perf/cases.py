"""The work that is timed: frames of soft-body scenes through the public entry points.

A program that uses this framework builds scenes from a mesh and a material, and then, frame
after frame, steps them and reads the state back.  A case is one such program: a single scene
(VBD, XPBD or explicit) stepped by `Scene.step` and read by `get_position` / `get_velocity`,
a batch of scenes stepped by `Batch.step` and read by `Batch.get_state`, or the per-frame
quantities a recorder writes (stress, volume change, energy) of a pose the program sets.

One pass is one frame; the next pass carries the simulation on.  Meshes are beams of hex
cells (cut into six tetrahedra for the tetrahedral elements), the shape that the framework's
own workloads have.  Inputs come from the seed: initial velocities, Young moduli, Poisson
ratios, poses.

`exact` restates the frame in 64 bits with torch and numpy alone: the colourings, the three
solvers and the recorded quantities.
"""
import heapq
import math
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import octopusengine_b200 as ob

P1, Q1, P2, P3, Q2 = ob.TETRA, ob.HEXA, ob.TETRA10, ob.TETRA20, ob.HEXA27
ELEMENT = {"P1": P1, "Q1": Q1, "P2": P2, "P3": P3, "Q2": Q2}
MATERIAL = {"NH": ob.NEOHOOKE, "SNH": ob.STABLE_NEOHOOKE, "StVK": ob.STVK}
NODES = {"P1": 4, "Q1": 8, "P2": 10, "P3": 20, "Q2": 27}
POINTS = {"P1": 1, "Q1": 8, "P2": 4, "P3": 11, "Q2": 27}
GRAVITY = (0.0, 0.0, -9.81)


def listed():
    def scene(name, solver, element, cells, **kw):
        c = dict(name=name, kind="scene", solver=solver, element=element, nx=cells[0], ny=cells[1], nz=cells[2],
                 edge=1.0 / 16, material="SNH", young=1e6, poisson=0.45, density=1000.0, v0=0.05, damping=0.0,
                 rho=0.0, iterations=10, substeps=1, dt=1.0 / 60, mixed=False, capture=False, spread=0.0)
        c.update(kw)
        return c

    return [
        # the smallest scene: a prop of 192 elements stepped once per frame, all latency
        scene("vbd_p1_8x2x2", "vbd", "P1", (8, 2, 2), edge=0.125, young=1e5, iterations=20, dt=0.01),
        # an ordinary prop on an odd grid whose cell edge is not a power of two, with Chebyshev
        # acceleration, damping and the mixed precision
        scene("vbd_q1_29x7x11", "vbd", "Q1", (29, 7, 11), edge=0.03, young=3e5, poisson=0.4, damping=1e-4, rho=0.9,
              substeps=2, mixed=True),
        # linear tetrahedra at the size of the reference's small-step beams
        scene("vbd_p1_64x16x16", "vbd", "P1", (64, 16, 16), substeps=2),
        # the quadratic beam of the single-scene workload: 98,304 P2 elements, 5 sub-steps of 10
        scene("vbd_p2_64x16x16", "vbd", "P2", (64, 16, 16), poisson=0.49, density=1100.0, substeps=5),
        # cubic tetrahedra with a Young modulus per element
        scene("vbd_p3_12x12x12", "vbd", "P3", (12, 12, 12), young=1e5, spread=1.0, substeps=2, mixed=True),
        # quadratic hexahedra at the size of the reference's small-step beams
        scene("vbd_q2_32x8x8", "vbd", "Q2", (32, 8, 8), substeps=2),
        # XPBD, frames replayed from a graph: the quadratic beam, and linear tetrahedra with the
        # small steps that XPBD is used with (moving at speeds that strain the elements by a
        # percent: below that its constraints are at the rounding of 32 bits)
        scene("xpbd_p2_64x16x16", "xpbd", "P2", (64, 16, 16), poisson=0.49, density=1100.0, v0=0.5, substeps=5,
              capture=True),
        scene("xpbd_p1_64x16x16", "xpbd", "P1", (64, 16, 16), v0=0.5, substeps=10, capture=True),
        # explicit integration of the quadratic beam, 100 steps of 10 us replayed from a graph
        scene("explicit_p2_64x16x16", "explicit", "P2", (64, 16, 16), poisson=0.49, density=1100.0, substeps=100,
              dt=1e-3, capture=True),
        # many independent objects in one batch: P1, Q1 and P2 beams of mixed sizes and materials
        dict(name="batch_vbd_16", kind="batch", solver="vbd", scenes=16, max_nx=96, max_ny=24, iterations=20,
             substeps=4, dt=1.0 / 60),
        dict(name="batch_xpbd_16", kind="batch", solver="xpbd", scenes=16, max_nx=48, max_ny=12, iterations=1,
             substeps=5, dt=1.0 / 60),
        # what a recorder writes of a pose: von Mises stress, volume change and energies
        dict(name="record_p2_64x16x16", kind="record", solver="vbd", element="P2", nx=64, ny=16, nz=16, edge=1.0 / 16,
             material="SNH", young=1e6, poisson=0.49, density=1100.0, damping=0.0, rho=0.0, iterations=1, spread=0.0,
             v0=0.0, mixed=False),
    ]


# Most cells per element type: the listed sizes.
MOST_CELLS = {"P1": 16384, "Q1": 16384, "P2": 16384, "P3": 1728, "Q2": 2048}


def _beam(rng, most):
    """Cells of a beam with between 8 and `most` cells, log-uniform, up to four times as long as wide."""
    n = math.exp(rng.uniform(math.log(8), math.log(most)))
    a, b = rng.uniform(1, 4), rng.uniform(0.7, 1.4)
    w = (n / a) ** (1 / 3)
    ny, nz = max(1, int(w * b)), max(1, int(w / b))
    return max(2, min(96, int(n / (ny * nz)))), ny, nz


def draw(rng):
    what = rng.choice(("vbd", "vbd", "vbd", "xpbd", "explicit", "batch", "record"))
    if what == "batch":
        solver = rng.choice(("vbd", "xpbd"))
        return dict(kind="batch", solver=solver, scenes=rng.randint(2, 16 if solver == "vbd" else 8),
                    max_nx=rng.randint(8, 64), max_ny=rng.randint(4, 16), iterations=rng.randint(5, 20),
                    substeps=rng.randint(1, 4), dt=1.0 / 60)
    element = rng.choice(("P1", "Q1", "P2", "P3", "Q2") if what in ("vbd", "record") else ("P1", "Q1", "P2"))
    nx, ny, nz = _beam(rng, MOST_CELLS[element])
    c = dict(kind="scene", solver=what, element=element, nx=nx, ny=ny, nz=nz, edge=rng.uniform(0.03, 0.125),
             material=rng.choice(("SNH", "SNH", "NH")), young=math.exp(rng.uniform(math.log(1e5), math.log(3e6))),
             poisson=rng.uniform(0.3, 0.49), density=1000.0, v0=0.05, damping=0.0, rho=0.0, iterations=1,
             substeps=1, dt=1.0 / 60, mixed=rng.random() < 0.5, capture=rng.random() < 0.5, spread=0.0)
    if what == "vbd":
        c.update(iterations=rng.randint(5, 20), substeps=rng.randint(1, 3), rho=rng.choice((0.0, 0.0, 0.9)),
                 damping=rng.choice((0.0, 0.0, 1e-4)), spread=rng.choice((0.0, 0.0, 1.0)))
    elif what == "xpbd":
        c.update(substeps=rng.randint(2, 10), mixed=False, v0=0.5)
    elif what == "explicit":
        c.update(substeps=rng.randint(20, 100), edge=rng.uniform(0.05, 0.125), young=1e6, material=rng.choice(("SNH", "NH", "StVK")),
                 damping=0.0)
        c["dt"] = 1e-5 * c["substeps"]
    else:
        c.update(kind="record", solver="vbd", v0=0.0, mixed=False)
        for k in ("substeps", "dt", "capture"):
            del c[k]
    return c


# ---------------------------------------------------------------------------- inputs
# Local nodes of each element as lattice points of its corners: (weights over the corners).
_HEX = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1),
        (0, -1, -1), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0),
        (0, -1, 1), (1, 0, 1), (0, 1, 1), (-1, 0, 1), (0, 0, -1), (0, -1, 0), (1, 0, 0), (0, 1, 0),
        (-1, 0, 0), (0, 0, 1), (0, 0, 0)]
_P2_EDGES = [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]
_P3_EDGES = [(0, 1), (1, 0), (1, 2), (2, 1), (2, 0), (0, 2), (0, 3), (3, 0), (1, 3), (3, 1), (2, 3), (3, 2)]
_P3_FACES = [(0, 1, 3), (1, 2, 3), (0, 2, 3), (0, 1, 2)]
_TETS = np.array([[0, 4, 6, 5], [3, 6, 2, 0], [0, 4, 7, 6], [3, 6, 0, 7], [2, 0, 6, 1], [6, 0, 5, 1]])


def _corner_weights(element):
    """Integer weights over the element's corners of each local node, and their sum."""
    w = np.zeros((NODES[element], 4 if element[0] == "P" else 8), np.int64)
    w[:w.shape[1]] = np.eye(w.shape[1], dtype=np.int64)
    if element == "P2":
        w *= 2
        for k, (i, j) in enumerate(_P2_EDGES):
            w[4 + k, [i, j]] = 1
        return w, 2
    if element == "P3":
        w *= 3
        for k, (i, j) in enumerate(_P3_EDGES):
            w[4 + k, i], w[4 + k, j] = 2, 1
        for k, f in enumerate(_P3_FACES):
            w[16 + k, list(f)] = 1
        return w, 3
    if element == "Q2":
        for n, p in enumerate(_HEX):
            for c in range(8):
                w[n, c] = np.prod([2 if q == s else 1 if q == 0 else 0 for q, s in zip(p, _HEX[c])])
        return w, 8
    return w, 1


def beam(element, nx, ny, nz, edge):
    """(X, T): a beam of nx x ny x nz cubic cells of the given edge, x along its length."""
    Nx, Ny = nx + 1, ny + 1
    z, y, x = (a.reshape(-1) for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    step = np.array([(0, 0, 0), (1, 0, 0), (1, 0, 1), (0, 0, 1), (0, 1, 0), (1, 1, 0), (1, 1, 1), (0, 1, 1)])
    at = np.stack([x, y, z], 1)[:, None, :] + step[None]                        # cell corners on the grid
    corner = at if element[0] == "Q" else at[:, _TETS].reshape(-1, 4, 3)
    w, k = _corner_weights(element)
    at = np.einsum("ecd,nc->end", corner, w) // (k // {1: 1, 2: 2, 3: 3, 8: 2}[k])  # on a grid k times finer
    fine = {1: 1, 2: 2, 3: 3, 8: 2}[k]
    nc = corner.shape[1]
    grid = corner[..., 0] + Nx * (corner[..., 1] + Ny * corner[..., 2])
    T = np.empty(at.shape[:2], np.int64)
    T[:, :nc] = grid
    gz, gy, gx = (a.reshape(-1) for a in np.meshgrid(np.arange(nz + 1), np.arange(Ny), np.arange(Nx), indexing="ij"))
    X = [np.stack([gx, gy, gz], 1) * fine]
    if at.shape[1] > nc:   # the other nodes in the order in which the elements meet them
        extra = at[:, nc:].reshape(-1, 3)
        key = extra[:, 0] + (fine * Nx + 1) * (extra[:, 1] + (fine * Ny + 1) * extra[:, 2])
        _, first, inverse = np.unique(key, return_index=True, return_inverse=True)
        rank = np.empty(len(first), np.int64)
        rank[np.argsort(first)] = np.arange(len(first))
        T[:, nc:] = (len(X[0]) + rank[inverse.reshape(-1)]).reshape(len(at), -1)
        X.append(extra[np.sort(first)])
    return (np.concatenate(X) * (edge / fine)).astype(np.float32), T.astype(np.int32)


def _members(case, seed):
    """The single-scene cases of a batch: beams of mixed element, size and material."""
    r, got = random.Random(9000 + seed), []
    shape = random.Random(case["scenes"] * 1000 + case["max_nx"])   # the sizes belong to the case, not to the seed
    for k in range(case["scenes"]):
        nx, ny, nz = shape.randint(4, case["max_nx"]), shape.randint(2, case["max_ny"]), shape.randint(2, case["max_ny"])
        got.append(dict(element=shape.choice(("P1", "P2", "Q1")), nx=nx, ny=ny, nz=nz, edge=1.0 / 16, material="SNH",
                        young=math.exp(r.uniform(math.log(1e5), math.log(1e7))), poisson=r.uniform(0.3, 0.49),
                        density=1000.0, v0=0.5 if case["solver"] == "xpbd" else 0.02, damping=0.0, rho=0.0, iterations=case["iterations"],
                        solver=case["solver"], mixed=True, spread=0.0))
    return got


def _inputs(c, seed):
    """Mesh, fixed nodes, initial velocities and Young moduli of one scene."""
    X, T = beam(c["element"], c["nx"], c["ny"], c["nz"], c["edge"])
    rng = np.random.default_rng(seed)
    fixed = np.nonzero(X[:, 0] < 1e-4)[0].astype(np.int32)
    young = np.full(len(T), c["young"], np.float32)
    if c["spread"]:
        young = (young * np.exp(rng.uniform(-c["spread"], c["spread"], len(T)))).astype(np.float32)
    v0 = rng.normal(0.0, c["v0"], X.shape).astype(np.float32) if c["v0"] else None
    return X, T, fixed, young, v0


def _pose(X, seed):
    """A smooth bent and stretched pose of the rest positions."""
    r = np.random.default_rng(seed)
    x = X.astype(np.float64) / max(float(np.abs(X).max()), 1e-9)
    size = float(X.max())
    a = r.uniform(0.01, 0.03, (3, 3)) * size
    f = r.uniform(1.0, 3.0, (3, 3))
    d = sum(a[k] * np.sin(x[:, k:k + 1] * f[k]) for k in range(3))
    return (X + d).astype(np.float32)


def _scene(ctx, c, X, T, fixed, young, v0):
    kw = dict(solver={"vbd": ob.SOLVER_VBD, "xpbd": ob.SOLVER_XPBD, "explicit": ob.SOLVER_EXPLICIT}[c["solver"]],
              material=MATERIAL[c["material"]], young=c["young"], poisson=c["poisson"], density=c["density"],
              gravity=GRAVITY, iterations=c["iterations"], damping=c["damping"], rho=c["rho"], fixed_ids=fixed,
              precision=ob.PREC_MIXED if c["mixed"] else ob.PREC_PLAIN)
    if c["spread"]:
        kw["young_per_element"] = young
    if v0 is not None:
        kw["initial_velocity"] = v0
    return ob.Scene(ctx, ELEMENT[c["element"]], X, T, **kw)


def prepare(case, seed):
    ctx = ob.Context(0)
    if case["kind"] == "batch":
        def build(k):
            return _scene(ctx, members[k], *_inputs(members[k], seed * 100 + k))
        members = _members(case, seed)
        with ThreadPoolExecutor(8) as pool:
            scenes = list(pool.map(build, range(len(members))))
        batch = ob.Batch(ctx, scenes)
        host = torch.empty(batch.state_size, dtype=torch.float32, pin_memory=True).numpy()
        cuts = np.cumsum([6 * s.n_nodes for s in scenes])[:-1]
        return dict(case=case, ctx=ctx, batch=batch, host=host, cuts=cuts)
    X, T, fixed, young, v0 = _inputs(case, seed)
    s = _scene(ctx, case, X, T, fixed, young, v0)
    if case["kind"] == "record":
        return dict(case=case, ctx=ctx, scene=s, pose=_pose(X, seed))
    if case["capture"]:
        s.set_capture(True)
    return dict(case=case, ctx=ctx, scene=s)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].step(case["dt"], case["substeps"])
        state["batch"].get_state(state["host"])
        return np.split(state["host"], state["cuts"])   # per scene: displacements, then velocities
    s = state["scene"]
    if case["kind"] == "record":
        s.set_position(state["pose"])
        return {"stress": s.element_data(ob.DIAG_STRESS), "volume": s.element_data(ob.DIAG_VOLUME_DIFF), "energy": s.energy()}
    s.step(case["dt"], case["substeps"])
    return {"p": s.get_position(), "v": s.get_velocity()}


def _counts(c):
    cells = c["nx"] * c["ny"] * c["nz"]
    grid = lambda k: (k * c["nx"] + 1) * (k * c["ny"] + 1) * (k * c["nz"] + 1)  # noqa: E731
    n = {"P1": grid(1), "Q1": grid(1), "P2": grid(2), "P3": grid(3), "Q2": grid(2)}[c["element"]]
    return n, cells * (6 if c["element"][0] == "P" else 1)


def work(case):
    """Bytes: the state in and out, masses, topology and one material record per element, once a
    pass.  Flops: per (node, element, point) of a VBD iteration, or per (element, point) of the
    other solvers, the deformation gradient, stress and (VBD) Hessian in closed form."""
    bytes_ = flops = 0.0
    for c in _members(case, 0) if case["kind"] == "batch" else [case]:
        n, e = _counts(c)
        ne, nq = NODES[c["element"]], POINTS[c["element"]]
        bytes_ += n * (2 * 24 + 16) + e * (4 * ne + 8)
        jx = {"P1": 18, "Q1": 65, "P2": 44, "P3": 360, "Q2": 150}[c["element"]]   # du/dxi at one point
        steps = case.get("substeps", 1)
        if case["kind"] == "record":
            flops += e * nq * (2 * jx + 400.0)
        elif c["solver"] == "vbd":
            flops += float(steps) * c["iterations"] * e * ne * nq * (jx + 170.0)
        else:
            flops += float(steps) * (2 if c["solver"] == "xpbd" else 1) * e * nq * (jx + 150.0 + 18 * ne)
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------- 64 bits
_T20 = [(0.040490506727590428, 0.013560701879802881, 0.77125473269537614, 0.039251090924839957),
        (0.75250850700965499, 0.068099370938206658, 0.097987203649279112, 0.055273369155936898),
        (0.067223294893383398, 0.035183929773598716, 0.15636389323939529, 0.055393798871576368),
        (0.41926631387951302, 0.047781435559086663, 0.47961101102565507, 0.059933185146559528),
        (0.45076587609127683, 0.059456616299433829, 0.056824017127933668, 0.069469965937635367),
        (0.12941137378891041, 0.33019041483746447, 0.0023910074574393647, 0.076162715245558357),
        (0.12154199133392780, 0.30649398842969028, 0.56297276014304609, 0.079426680068025307),
        (0.097204644587583267, 0.68439041545304002, 0.11180076739738309, 0.10646803415549010),
        (0.029569495206479612, 0.31790356021339461, 0.32329398483747895, 0.11023423242849766),
        (0.43271023904776856, 0.35382323920929709, 0.10962240533194123, 0.15497611601624608),
        (0.24027666492807262, 0.12680172591539202, 0.32847320672203845, 0.19341081204963445)]
_DL = np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], np.float64)


def _shape(element):
    """(dN [points, nodes, 3], weights) of an element."""
    if element[0] == "Q":
        if element == "Q1":
            pts, w = [np.array(p) / math.sqrt(3) for p in _HEX[:8]], [1.0] * 8
        else:
            pts = [np.array(p) * math.sqrt(0.6) for p in _HEX]
            w = [np.prod([8 / 9 if q == 0 else 5 / 9 for q in p]) for p in _HEX]

        def one(node, s):   # 1-D basis and derivative
            if element == "Q1":
                return (1 + node * s) / 2, node / 2
            return (s * (s + node) / 2, s + node / 2) if node else (1 - s * s, -2 * s)
        dN = np.zeros((len(pts), NODES[element], 3))
        for q, p in enumerate(pts):
            for i in range(NODES[element]):
                b = [one(_HEX[i][k], p[k]) for k in range(3)]
                for k in range(3):
                    dN[q, i, k] = np.prod([b[m][1 if m == k else 0] for m in range(3)])
        return dN, np.array(w)
    if element == "P1":
        pts, w = [(0.25, 0.25, 0.25)], [1 / 6]
    elif element == "P2":
        a, b = (5 - math.sqrt(5)) / 20, (5 + 3 * math.sqrt(5)) / 20
        pts, w = [(b, a, a), (a, b, a), (a, a, b), (a, a, a)], [1 / 24] * 4
    else:
        pts, w = [p[:3] for p in _T20], [p[3] / 6 for p in _T20]
    dN = np.zeros((len(pts), NODES[element], 3))
    for q, (x, y, z) in enumerate(pts):
        L = (1 - x - y - z, x, y, z)
        for i in range(4):
            dN[q, i] = _DL[i] * {"P1": 1.0, "P2": 4 * L[i] - 1, "P3": (27 * L[i] ** 2 - 18 * L[i] + 2) / 2}[element]
        if element == "P2":
            for k, (i, j) in enumerate(_P2_EDGES):
                dN[q, 4 + k] = 4 * (L[j] * _DL[i] + L[i] * _DL[j])
        if element == "P3":
            for k, (i, j) in enumerate(_P3_EDGES):
                dN[q, 4 + k] = 4.5 * (L[j] * (6 * L[i] - 1) * _DL[i] + L[i] * (3 * L[i] - 1) * _DL[j])
            for k, (i, j, m) in enumerate(_P3_FACES):
                dN[q, 16 + k] = 27 * (L[j] * L[m] * _DL[i] + L[i] * L[m] * _DL[j] + L[i] * L[j] * _DL[m])
    return dN, np.array(w)


def _graph(pairs, n):
    """Neighbours and their multiplicities per row, as lists, from directed (row, neighbour) keys row * n + neighbour."""
    key, mult = np.unique(pairs, return_counts=True)
    off = np.searchsorted(key, np.arange(n + 1) * n).tolist()
    nbr, mult = (key % n).tolist(), mult.tolist()
    return [nbr[off[i]:off[i + 1]] for i in range(n)], [mult[off[i]:off[i + 1]] for i in range(n)]


def _vertex_graph(T, n):
    T = T.astype(np.int64)
    ne = T.shape[1]
    return _graph(np.concatenate([T[:, i] * n + T[:, j] for i in range(ne) for j in range(ne) if i != j]), n)


def _element_graph(T, n):
    """Elements that share a node, once for each node that they share."""
    e, ne = T.shape
    order = np.argsort(T.reshape(-1), kind="stable")
    own = order // ne
    count = np.bincount(T.reshape(-1), minlength=n)
    start = np.cumsum(count) - count
    rows, cols = [], []
    for k in range(int(count.max())):
        node = np.nonzero(count > k)[0]
        a = own[start[node] + k]
        reps = count[node]
        base = np.repeat(start[node], reps) + np.arange(reps.sum()) - np.repeat(np.cumsum(reps) - reps, reps)
        rows.append(np.repeat(a, reps))
        cols.append(own[base])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    keep = rows != cols
    return _graph(rows[keep] * np.int64(e) + cols[keep], e)


def _dsat(nbr, mult):
    """Largest (saturation, remaining degree, index) first, smallest free colour."""
    n = len(nbr)
    degree = [sum(m) for m in mult]
    color, seen, sat = [-1] * n, [0] * n, [0] * n
    heap = [-((degree[v] << 27) | v) for v in range(n)]
    current = list(heap)
    heapq.heapify(heap)
    low = (1 << 27) - 1
    while heap:
        top = heapq.heappop(heap)
        v = -top & low
        if color[v] >= 0 or current[v] != top:
            continue
        c, s = 0, seen[v]
        while s >> c & 1:
            c += 1
        color[v] = c
        bit = 1 << c
        for w, m in zip(nbr[v], mult[v]):
            if color[w] >= 0:
                continue
            if not seen[w] & bit:
                seen[w] |= bit
                sat[w] += 1
            degree[w] -= m
            k = -((sat[w] << 51) | (degree[w] << 27) | w)
            current[w] = k
            heapq.heappush(heap, k)
    return np.array(color)


def _smallest_last(nbr, mult):
    """Greedy colouring, the row of least remaining degree coloured last."""
    n = len(nbr)
    degree = [sum(m) for m in mult]
    heap = [(degree[v] << 27) | v for v in range(n)]
    heapq.heapify(heap)
    gone, order, low = [False] * n, [], (1 << 27) - 1
    while heap:
        v = heapq.heappop(heap) & low
        if gone[v]:
            continue
        gone[v] = True
        order.append(v)
        for w, m in zip(nbr[v], mult[v]):
            if not gone[w]:
                degree[w] -= m
                heapq.heappush(heap, (degree[w] << 27) | w)
    color = [-1] * n
    for v in reversed(order):
        used = 0
        for w in nbr[v]:
            if color[w] >= 0:
                used |= 1 << color[w]
        c = 0
        while used >> c & 1:
            c += 1
        color[v] = c
    return np.array(color)


class _Exact:
    """One scene in 64 bits."""

    def __init__(self, c, seed):
        self.c = c
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        X, T, fixed, young, v0 = _inputs(c, seed)
        self.X32, self.T = X, T
        put = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        f64 = lambda a: put(np.asarray(a, np.float64))  # noqa: E731
        self.put = put
        dN, w = _shape(c["element"])
        self.dN, self.t = f64(dN), put(T.astype(np.int64))
        self.x = f64(X)
        J = torch.einsum("eni,qnk->eqik", self.x[self.t], self.dN)
        self.inv, self.V = torch.linalg.inv(J), torch.linalg.det(J).abs() * f64(w)
        Y, nu = young.astype(np.float64), float(np.float32(c["poisson"]))
        self.lam = f64((Y * nu / ((1 + nu) * (1 - 2 * nu))).astype(np.float32))
        self.mu = f64((Y / (2 * (1 + nu))).astype(np.float32))
        self.m = torch.zeros(len(X), dtype=torch.float64, device=self.dev)
        share = self.V.sum(1) * c["density"] / T.shape[1]
        self.m.index_add_(0, self.t.reshape(-1), share[:, None].expand(-1, T.shape[1]).reshape(-1))
        self.u = torch.zeros_like(self.x)
        self.v = f64(v0) if v0 is not None else torch.zeros_like(self.x)
        self.fixed = put(fixed.astype(np.int64))
        self.free = torch.ones(len(X), dtype=torch.bool, device=self.dev)
        self.g = f64(np.array(GRAVITY, np.float32))
        self.eye = torch.eye(3, dtype=torch.float64, device=self.dev)

    def F(self, e):
        return self.eye + torch.einsum("eni,qnk->eqik", self.u[self.t[e]], self.dN) @ self.inv[e]

    def cof(self, F):
        a, b, c = F.unbind(-1)
        return torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -1)

    def stress(self, F, lam, mu):
        """First Piola-Kirchhoff stress and the cofactor."""
        K = self.cof(F)
        det = (F[..., 0] * K[..., 0]).sum(-1)[..., None, None]
        if self.c["material"] == "StVK":
            E = (F.transpose(-1, -2) @ F - self.eye) / 2
            tr = E.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
            return lam * tr * F + 2 * mu * (F @ E), K
        s = lam * (det - 1) - (mu if self.c["material"] == "SNH" else 0)
        return mu * F + s * K, K

    def fix(self):
        self.u[self.fixed] = 0.0
        self.v[self.fixed] = 0.0
        self.free[self.fixed] = False

    # --- VBD: Gauss-Seidel over the colours of the vertex graph
    def vbd_plan(self):
        color = _dsat(*_vertex_graph(self.T, len(self.X32)))
        flat = self.T.reshape(-1)
        ne = self.T.shape[1]
        plan = []
        for c in range(color.max() + 1):
            at = np.nonzero(color[flat] == c)[0]
            ids, seg = np.unique(flat[at], return_inverse=True)
            plan.append(tuple(self.put(a.astype(np.int64)) for a in (ids, seg.reshape(-1), at // ne, at % ne)))
        return plan

    def vbd_color(self, ids, seg, e, r, y, u0, h):
        out = torch.zeros((len(ids), 3), dtype=torch.float64, device=self.dev)
        H = torch.zeros((len(ids), 3, 3), dtype=torch.float64, device=self.dev)
        for a in range(0, len(e), 1 << 18):
            b = slice(a, a + (1 << 18))
            F = self.F(e[b])
            lam, mu = self.lam[e[b]][:, None, None, None], self.mu[e[b]][:, None, None, None]
            P, K = self.stress(F, lam, mu)
            g = torch.einsum("eqk,eqkb->eqb", self.dN[:, r[b]].transpose(0, 1), self.inv[e[b]])[..., None]
            V = self.V[e[b]][..., None, None]
            k = K @ g
            out.index_add_(0, seg[b], -(V * (P @ g))[..., 0].sum(1))
            gg = (g * g).sum(-2, keepdim=True)
            H.index_add_(0, seg[b], (V * (mu * gg * self.eye + lam * (k @ k.transpose(-1, -2)))).sum(1))
        kd = float(np.float32(self.c["damping"])) / h
        d = (self.u[ids] - u0[ids])[..., None]
        out -= kd * (H @ d)[..., 0]
        H *= 1 + kd
        mh = self.m[ids][:, None] / h ** 2
        out -= mh * (self.u[ids] - y[ids])
        H += mh[..., None] * self.eye
        step = torch.linalg.solve(H, out)
        self.u[ids] += torch.where(self.free[ids][:, None], step, torch.zeros_like(step))

    def vbd(self, dt, substeps):
        plan, rho, c = self.vbd_plan(), float(np.float32(self.c["rho"])), self.c
        h = float(np.float32(np.float32(dt) / np.float32(substeps)))
        last = self.u - self.v * h
        for _ in range(substeps):
            u0 = self.u.clone()
            y = self.u + (self.u - last) + self.g * h * h
            self.u = y.clone()
            before, omega = [u0], 1.0
            for j in range(c["iterations"]):
                for part in plan:
                    self.vbd_color(*part, y, u0, h)
                self.fix()
                if rho:
                    if j == 1:
                        omega = 2 / (2 - rho * rho)
                    elif j > 1:
                        omega = 4 / (4 - rho * rho * omega)
                        self.u = before[-2] + omega * (self.u - before[-2])
                    before.append(self.u.clone())
            last = u0
            self.v = (self.u - u0) / h

    # --- XPBD: two constraints per element, colours of the element graph
    def xpbd(self, dt, substeps):
        c = self.c
        color = _smallest_last(*_element_graph(self.T, len(self.X32)))
        plan = [self.put(np.nonzero(color == k)[0]) for k in range(color.max() + 1)]
        h = float(np.float32(np.float32(dt) / np.float32(substeps)))
        w = 1 / self.m
        for _ in range(substeps):
            u0 = self.u.clone()
            self.v = self.v + self.g * h
            self.u = self.u + self.v * h
            for e in plan:
                t = self.t[e]
                for m in (0, 1):
                    k = (self.lam if m == 0 else self.mu)[e]
                    F = self.F(e)
                    K = self.cof(F)
                    det = (F[..., 0] * K[..., 0]).sum(-1)
                    n2 = (F * F).sum((-1, -2)) - 3
                    if m == 0:
                        d = det - (1 + (self.mu / self.lam)[e][:, None] if c["material"] == "NH" else 1.0)
                        C, P = d * d, 2 * d[..., None, None] * K
                    elif c["material"] == "NH":
                        C, P = n2, 2 * F
                    else:
                        C, P = n2 - 2 * (det - 1), 2 * F - 2 * K
                    V = self.V[e]
                    C = (C * V).sum(1)
                    grad = torch.einsum("eqik,qnk->eni", (P @ self.inv[e].transpose(-1, -2)) * V[..., None, None], self.dN)
                    s2 = ((grad * grad).sum(-1) * w[t]).sum(1)
                    if c["element"] == "P1":   # normalised update; fixed nodes stay
                        C = C.abs().sqrt()
                        grad = grad * torch.where(C < 1e-12, torch.zeros_like(C), 1 / (2 * C))[:, None, None]
                        s2 = ((grad * grad).sum(-1) * w[t]).sum(1)
                        f = (-C / (s2 + 1 / (k * h * h)))[:, None] * w[t] * self.free[t]
                    else:
                        f = torch.where(C < 1e-12, torch.zeros_like(C), -2 * C / (s2 + 4 * C / (k * h * h)))[:, None] * w[t]
                    self.u[t] = self.u[t] + f[..., None] * grad
            self.fix()
            self.v = (self.u - u0) / h

    def explicit(self, dt, substeps):
        h = float(np.float32(np.float32(dt) / np.float32(substeps)))
        every = slice(None)
        for _ in range(substeps):
            P, _ = self.stress(self.F(every), self.lam[:, None, None, None], self.mu[:, None, None, None])
            f = torch.einsum("eqik,qnk->eni", (P @ self.inv.transpose(-1, -2)) * self.V[..., None, None], self.dN)
            a = torch.zeros_like(self.u).index_add_(0, self.t.reshape(-1), -f.reshape(-1, 3)) / self.m[:, None]
            self.v = self.v + (self.g + a) * h
            self.u = self.u + self.v * h
            self.fix()

    def step(self, dt, substeps):
        getattr(self, self.c["solver"])(dt, substeps)

    def record(self, pose):
        X = self.X32
        u = pose - X
        p = torch.as_tensor(np.asarray(X + u, np.float64), device=self.dev)   # in the 32 bits that the scene holds
        J = torch.einsum("eni,qnk->eqik", p[self.t], self.dN)
        F = J @ self.inv
        lam, mu = self.lam[:, None, None, None], self.mu[:, None, None, None]
        P, _ = self.stress(F, lam, mu)
        S = P @ F.transpose(-1, -2) / torch.linalg.det(F)[..., None, None]
        d = [S[..., 0, 0] - S[..., 1, 1], S[..., 1, 1] - S[..., 2, 2], S[..., 0, 0] - S[..., 2, 2]]
        shear = S[..., 1, 0] ** 2 + S[..., 2, 1] ** 2 + S[..., 2, 0] ** 2
        vm = (0.5 * (d[0] ** 2 + d[1] ** 2 + d[2] ** 2) + 3 * shear).sqrt()
        detJ = torch.linalg.det(J).abs()
        w = torch.as_tensor(_shape(self.c["element"])[1], device=self.dev)
        F = self.eye + torch.einsum("eni,qnk->eqik", torch.as_tensor(u.astype(np.float64), device=self.dev)[self.t], self.dN) @ self.inv
        alpha = 1 + self.mu / self.lam if self.c["material"] == "SNH" else torch.ones_like(self.mu)
        psi = 0.5 * mu[..., 0, 0] * ((F * F).sum((-1, -2)) - 3) + 0.5 * lam[..., 0, 0] * (torch.linalg.det(F) - alpha[:, None]) ** 2
        elastic = float((psi * self.V).sum())
        grav = -float((self.m[:, None] * self.g * p).sum())
        return {"stress": (vm * self.V).sum(1).cpu().numpy(), "volume": (detJ * w - self.V).sum(1).cpu().numpy(),
                "energy": np.array([0.0, elastic, grav, elastic + grav])}


def exact(case, seed):
    if case["kind"] == "batch":
        got = []
        for k, c in enumerate(_members(case, seed)):
            s = _Exact(c, seed * 100 + k)
            s.step(case["dt"], case["substeps"])
            got.append(torch.cat([s.u.reshape(-1), s.v.reshape(-1)]).cpu().numpy())
        return got
    s = _Exact(case, seed)
    if case["kind"] == "record":
        return s.record(_pose(s.X32, seed))
    s.step(case["dt"], case["substeps"])
    return {"p": (s.x + s.u).cpu().numpy(), "v": s.v.cpu().numpy()}
