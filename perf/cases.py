"""What this framework is timed on: frames of every solver kind, the smoother's network and the diagnostics,
each through the calls that a user's program makes.

A frame pass is one turn of a simulation loop: move the tool, `step()`, read positions and contact flags back.
The state advances from pass to pass as it does in a program; the tool goes down and up again over a fixed
stroke, so that a long run stays in the regime of its first frames.  Meshes are built here (voxel meshes, six
Kuhn tets per hex, numbered as `box_mesh` numbers them), so that `exact` needs nothing of the package.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import multigridsoftbody_b200 as mg
from multigridsoftbody_b200.learned import MLP

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOOL_FRAMES = 28          # frames of one stroke of the tool, down and up again
LARGEST_HEXES = 24 * 240 * 24


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    beam = {"path": "frame", "shape": "beam", "nx": 12, "ny": 120, "nz": 12, "levels": 4, "precision": "fp32",
            "passes": 1, "sweeps": 2, "learned": False, "material": "uniform", "gravity": 0.0, "contact": "vertices",
            "split": 0, "dense": False}
    return [
        # An interactive scene of the reference's own size and solver, through its class (PDSolver): the smallest call.
        {"name": "reference_small", "path": "reference", "nx": 4, "ny": 14, "nz": 4, "iterations": 20, "mirror": True},
        # The reference's solver on the beam of its analysis (96,768 tets), through the general handle.
        {"name": "reference_beam", "path": "reference", "nx": 12, "ny": 112, "nz": 12, "iterations": 20,
         "mirror": False},
        # A small hanging beam without a tool, as a control loop or a unit of a larger program runs it.
        {**beam, "name": "beam_small", "nx": 4, "ny": 40, "nz": 4, "levels": 3, "gravity": -9.8, "contact": "none"},
        # The ordinary multigrid frame: 103,680 tets, FP32, the shape the solver picks by itself.
        {**beam, "name": "beam"},
        # The production form of the same scene: learned smoother, FP64 refinement, dense coarse operator.
        {**beam, "name": "beam_learned", "precision": "mixed", "passes": 2, "sweeps": 1, "learned": True, "split": 2,
         "dense": True},
        # The largest body: 829,440 tets, FP64 refinement, a material per tet.
        {**beam, "name": "beam_large", "nx": 24, "ny": 240, "nz": 24, "levels": 5, "precision": "mixed", "passes": 2,
         "material": "per_tet"},
        # Many uneven bodies with a tool each in one handle, as a training or planning service runs them.
        {"name": "batch", "path": "batch", "bodies": 128, "least": 2, "most": 8, "levels": 3, "sizes": 11},
        # An organ-like body: irregular surface and rows, gravity, contact with the surface triangles.
        {**beam, "name": "organ", "shape": "organ", "nx": 48, "ny": 24, "nz": 32, "levels": 5, "gravity": -9.8,
         "contact": "triangles"},
        # The reference's two-level schedule on its pair of meshes.
        {"name": "two_level", "path": "two_level", "nx": 12, "ny": 120, "nz": 12, "cx": 4, "cy": 40, "cz": 4,
         "iterations": 20},
        # Training the smoother's network on pairs that a solver generated.
        {"name": "train", "path": "train", "pairs": 200000, "steps": 100, "batch": 4096},
        # The network alone, on host features: checking a trained network on held-out pairs.
        {"name": "infer", "path": "infer", "rows": 100000},
        # What a viewer or a monitor asks for beside the frame: surface normals and the energies.
        {**beam, "name": "diagnostics", "path": "diagnostics"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _levels(nx, ny, nz):
    """Levels down to a coarsest grid of at most 150 nodes (its dense inverse stays in shared memory)."""
    dims, levels = [nx, ny, nz], 1
    while levels < 2 or (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1) > 150:
        dims = [max(1, (d + 1) // 2) for d in dims]
        levels += 1
    return levels


def _draw_box(rng, most):
    while True:
        nx, nz = _log_int(rng, 2, 24), _log_int(rng, 2, 24)
        ny = _log_int(rng, 8, 240)
        if 40 <= nx * ny * nz <= most and max(nx, nz) <= 3 * min(nx, nz) and ny >= max(nx, nz):
            return nx, ny, nz


def draw(rng):
    path = rng.choice(["reference", "reference", "frame", "frame", "frame", "frame", "organ", "batch", "two_level",
                       "train", "infer", "diagnostics"])
    if path == "reference":
        nx, ny, nz = _draw_box(rng, 20000)
        return {"path": path, "nx": nx, "ny": ny, "nz": nz, "iterations": rng.randint(5, 32),
                "mirror": rng.random() < 0.5}
    if path == "batch":
        least = rng.randint(2, 4)
        return {"path": path, "bodies": _log_int(rng, 3, 120), "least": least, "most": rng.randint(least, 8),
                "levels": 3, "sizes": rng.randint(1, 1 << 20)}
    if path == "two_level":
        c = rng.randint(2, 4)
        f = c * rng.randint(2, 3)
        return {"path": path, "nx": f, "ny": 10 * f, "nz": f, "cx": c, "cy": 10 * c, "cz": c,
                "iterations": rng.randint(5, 24)}
    if path == "train":
        return {"path": path, "pairs": _log_int(rng, 5000, 300000), "steps": rng.randint(40, 120),
                "batch": _log_int(rng, 500, 8192)}
    if path == "infer":
        return {"path": path, "rows": _log_int(rng, 50, 500000)}
    case = {"path": "frame", "shape": "beam", "precision": "fp32", "passes": 1, "sweeps": 2, "learned": False,
            "material": rng.choice(["uniform", "per_tet"]), "gravity": rng.choice([0.0, -9.8]),
            "contact": rng.choice(["vertices", "vertices", "vertices", "triangles", "none"]), "split": 0,
            "dense": False}
    if path == "organ":
        nx, ny, nz = rng.randint(12, 56), rng.randint(10, 28), rng.randint(12, 40)
        return {**case, "shape": "organ", "nx": nx, "ny": ny, "nz": nz, "levels": _levels(nx, ny, nz),
                "passes": rng.randint(1, 2)}
    nx, ny, nz = _draw_box(rng, LARGEST_HEXES // 3)
    case.update(nx=nx, ny=ny, nz=nz, levels=_levels(nx, ny, nz))
    if path == "diagnostics":
        return {**case, "path": path}
    form = rng.choice(["plain", "plain", "mixed", "learned"])
    case.update(passes=rng.randint(1, 2), sweeps=rng.randint(1, 2))
    if form != "plain":
        case["precision"] = "mixed"
    if form == "learned":
        case.update(learned=True, material="uniform", gravity=0.0)
    if case["levels"] > 2 and rng.random() < 0.4:   # the coarsest level but one as a dense operator
        case.update(split=case["levels"] - 2, dense=True)
        dims = [nx, ny, nz]
        for _ in range(case["split"]):
            dims = [max(1, (d + 1) // 2) for d in dims]
        if (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1) > 1000:   # above the operator's limit of rows
            case.update(split=0, dense=False)
    return case


# ---------------------------------------------------------------------------
# Meshes
# ---------------------------------------------------------------------------
def _kuhn(kept, lo, h):
    """Mesh of the kept voxels of a grid (kept[x, y, z]): positions, tets.  Vertices y slowest, then z, then x."""
    nx, ny, nz = kept.shape
    i, j, k = np.nonzero(kept)
    order = np.lexsort((i, k, j))
    cell = np.stack([i[order], j[order], k[order]], 1)
    corner = np.array([[c & 1, (c >> 1) & 1, (c >> 2) & 1] for c in range(8)])
    node = cell[:, None, :] + corner[None]
    key = (node[..., 1] * (nz + 1) + node[..., 2]) * (nx + 1) + node[..., 0]
    used, index = np.unique(key.reshape(-1), return_inverse=True)
    index = index.reshape(-1, 8)
    x, z, y = used % (nx + 1), (used // (nx + 1)) % (nz + 1), used // ((nx + 1) * (nz + 1))
    pos = np.stack([lo[0] + h[0] * x, lo[1] + h[1] * y, lo[2] + h[2] * z], 1).astype(np.float32)
    tets = []
    for perm, odd in (((0, 1, 2), 0), ((0, 2, 1), 1), ((1, 0, 2), 1), ((1, 2, 0), 0), ((2, 0, 1), 0), ((2, 1, 0), 1)):
        c, ids = [0, 0, 0], [0]
        for a in perm:
            c[a] = 1
            ids.append(c[0] + 2 * c[1] + 4 * c[2])
        if odd:
            ids[1], ids[2] = ids[2], ids[1]
        tets.append(index[:, ids])
    return pos, np.stack(tets, 1).reshape(-1, 4).astype(np.int32)


def _beam(nx, ny, nz, half=10.0):
    lo = (-1.0, -half, -1.0)
    h = (2.0 / nx, 2.0 * half / ny, 2.0 / nz)
    pos, tets = _kuhn(np.ones((nx, ny, nz), bool), lo, h)
    top = np.abs(pos[:, 1] - half) < 1e-4 * half
    pos[top, 1] = half
    return pos, tets, top.astype(np.uint8)


def _organ(nx, ny, nz):
    """The voxels of an ellipsoid of half axes 6, 3, 4 whose radius varies along it; the lower half lies on a table."""
    axes = np.array([6.0, 3.0, 4.0])
    g = np.stack(np.meshgrid(*[(np.arange(n) + 0.5) * 2.0 / n - 1.0 for n in (nx, ny, nz)], indexing="ij"), -1)
    wave = 0.9 + 0.1 * np.sin(5.0 * g[..., 0]) * np.cos(4.0 * g[..., 1] + 1.0) * np.cos(3.0 * g[..., 2])
    kept = (g * g).sum(-1) < wave
    pos, tets = _kuhn(kept, -axes, 2.0 * axes / np.array([nx, ny, nz]))
    return pos, tets, (pos[:, 2] < 0.0).astype(np.uint8)


def _body(case):
    """(positions, tets, fixed mask) of a single-body case."""
    if case.get("shape") == "organ":
        return _organ(case["nx"], case["ny"], case["nz"])
    return _beam(case["nx"], case["ny"], case["nz"])


def _batch(case):
    """Per body: (positions, tets, fixed, hexes per edge, E, nu), the same for every seed of a case."""
    rng = np.random.default_rng(case["sizes"])
    out, known = [], {}
    for n in rng.integers(case["least"], case["most"] + 1, size=case["bodies"]):
        n = int(n)
        if n not in known:
            known[n] = _beam(n, 10 * n, n, half=2.5 * n)
        E, nu = float(np.exp(rng.uniform(np.log(5e4), np.log(2e5)))), float(rng.uniform(0.25, 0.45))
        out.append((*known[n], n, np.float32(E), np.float32(nu)))
    return out


# ---------------------------------------------------------------------------
# Inputs of a seed
# ---------------------------------------------------------------------------
def _state(rest, fixed, rng):
    """A mildly deformed, moving state: a few smooth modes; the fixed vertices rest."""
    x = rest.astype(np.float64)
    size = float(np.ptp(x, axis=0).min())
    free = (1.0 - fixed)[:, None]
    u, v = np.zeros_like(x), np.zeros_like(x)
    for _ in range(3):
        k = rng.uniform(0.1, 0.6, 3)
        wave = np.sin(x @ k + rng.uniform(0, 6.28))[:, None]
        u += wave * rng.normal(0.0, 0.01, 3) * size
        v += wave * rng.normal(0.0, 0.1, 3) * size
    return (x + u * free).astype(np.float32), (v * free).astype(np.float32)


def _stroke(rng, start, depth, sigma):
    """Centres of the tool over one stroke from its middle: down, up by `depth` along z and down, with a tremor."""
    t = (np.arange(TOOL_FRAMES) + TOOL_FRAMES // 4) % TOOL_FRAMES / (TOOL_FRAMES / 2.0)
    z = np.where(t < 1.0, t, 2.0 - t)
    c = np.tile(np.asarray(start, np.float64), (TOOL_FRAMES, 1))
    c[:, 2] -= depth * z
    return c + rng.normal(0.0, sigma, c.shape)


def _frame_inputs(case, seed):
    """Body, state, material and tool of a frame case: everything `prepare` and `exact` take from the seed."""
    rng = np.random.default_rng(seed)
    if case["path"] == "batch":
        bodies = _batch(case)
        states = [_state(p, f, rng) for p, _, f, *_ in bodies]
        start = np.array([0.0, 0.0, 1.15]) + rng.uniform(-0.15, 0.15, (len(bodies), 3))
        tool = np.stack([_stroke(rng, s, 0.15, 0.01) for s in start], 1)         # [frame, body, 3]
        return bodies, states, tool, 2.0, 0.2
    rest, tets, fixed = _body(case)
    state = _state(rest, fixed, rng)
    if case["material"] == "per_tet":
        E = np.exp(rng.uniform(np.log(5e4), np.log(2e5), len(tets))).astype(np.float32)
    else:
        E = np.full(len(tets), 1e5, np.float32)
    nu = np.float32(0.45 if case["shape"] == "organ" else 0.3)
    top = 0.2 + float(rest[np.abs(rest[:, 1]) < 1.0, 2].max())
    start = (0.0, 0.0, top)
    tool = _stroke(rng, start, 0.25, 0.005)[:, None, :]
    return [(rest, tets, fixed, case["nx"], E, nu)], [state], tool, 4.0, 0.0 if case["contact"] == "none" else 0.3


def _sphere_path(case, seed):
    """Sphere centres (radius 0.8) pushed into the side of a beam and out again."""
    rng = np.random.default_rng(seed)
    c = np.zeros((TOOL_FRAMES, 3))
    t = (np.arange(TOOL_FRAMES) + TOOL_FRAMES // 4) % TOOL_FRAMES / (TOOL_FRAMES / 2.0)
    c[:, 0] = 1.6 - 0.25 * np.where(t < 1.0, t, 2.0 - t)
    c[:, 1] = -3.0 + rng.uniform(-1.0, 1.0)
    c[:, 2] = rng.uniform(-0.2, 0.2)
    return (c + rng.normal(0.0, 0.005, c.shape)).astype(np.float32)


def _reference_state(case, seed):
    rest, tets, fixed = _beam(case["nx"], case["ny"], case["nz"])
    return (rest, tets, fixed, *_state(rest, fixed, np.random.default_rng(seed + 1)))


def _pairs(rows, seed):
    """Features and targets of the network's ranges: unit residual directions, row constants, damped targets."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(rows, 6)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    x = np.empty((rows, 9), np.float32)
    x[:, 0:3], x[:, 6:9] = d[:, 0:3], d[:, 3:6]
    x[:, 3] = 1.0 + 0.3 * rng.random(rows, np.float32)
    x[:, 4] = np.where(rng.random(rows) < 0.05, 0.5 * rng.random(rows), 0.0)
    x[:, 5] = 0.7 + 0.6 * rng.random(rows, np.float32)
    t = 1.2 * x[:, 0:3] + 0.5 * x[:, 6:9] * x[:, 5:6] - 0.3 * x[:, 0:3] * x[:, 4:5]
    return x, t.astype(np.float32)


def _initial_parameters(seed):
    rng = np.random.default_rng(seed + 2)
    p = np.zeros(4995, np.float32)
    for at, out, inp in ((0, 64, 9), (640, 64, 64), (4800, 3, 64)):
        a = math.sqrt(6.0 / (inp + out))
        p[at:at + out * inp] = rng.uniform(-a, a, out * inp)
    return p


def _trained_parameters():
    return np.load(os.path.join(ROOT, "tests", "golden", "beam_smoother.npy"))


def _params(case):
    return mg.default_params(
        mg.SOLVER_MULTIGRID, levels=case["levels"], iterations=10,
        gravity=(0.0, 0.0, case["gravity"]) if case.get("shape") == "organ" else (0.0, case.get("gravity", 0.0), 0.0),
        precision=mg.PRECISION_MIXED if case.get("precision") == "mixed" else mg.PRECISION_FP32,
        refinement_passes=case.get("passes", 1), pre_sweeps=case.get("sweeps", 2), post_sweeps=case.get("sweeps", 2))


# ---------------------------------------------------------------------------
# What a program holds, and one pass
# ---------------------------------------------------------------------------
def _frame_arrays(n):
    """The host arrays that a program reads its frames into."""
    return {"positions": np.empty((n, 3), np.float32), "contact": np.empty(n, np.int32)}


def prepare(case, seed):
    path = case["path"]
    if path == "reference":
        rest, tets, fixed, x, v = _reference_state(case, seed)
        spheres = _sphere_path(case, seed)
        if case["mirror"]:
            s = mg.PDSolver()
            s.m_iterNum = case["iterations"]
            tool = mg.SphereCollider(spheres[0], 0.8)
            s.m_sphereColliders.append(tool)
            s.m_sphereFixers.append(mg.SphereFixer((0.0, 10.0, 0.0), 1.8))
            s.Init(rest, tets)
            s.solver.set_state(x, v)
            return {"path": path, "solver": s, "tool": tool, "spheres": spheres, "frame": 0}
        s = mg.Solver(mg.TetMesh(rest, tets), mg.default_params(mg.SOLVER_REFERENCE_JACOBI,
                                                                iterations=case["iterations"]))
        s.set_fixed(fixed)
        s.set_state(x, v)
        return {"path": path, "solver": s, "tool": None, "spheres": spheres, "frame": 0, **_frame_arrays(len(rest))}
    if path == "two_level":
        fine, coarse = _beam(case["nx"], case["ny"], case["nz"]), _beam(case["cx"], case["cy"], case["cz"])
        s = mg.TwoLevel(mg.TetMesh(*coarse[:2]), mg.TetMesh(*fine[:2]),
                        mg.default_params(mg.SOLVER_REFERENCE_JACOBI, iterations=case["iterations"]))
        s.set_fixed(coarse[2], fine[2])
        return {"path": path, "solver": s, "spheres": _sphere_path(case, seed), "frame": 0}
    if path in ("train", "infer"):
        net = MLP(device=0, seed=0)
        rows = case["pairs"] if path == "train" else case["rows"]
        x, t = _pairs(rows, seed)
        net.params = _initial_parameters(seed) if path == "train" else _trained_parameters()
        return {"path": path, "net": net, "x": x, "t": t, "case": dict(case), "seed": seed}
    bodies, states, tool, half, radius = _frame_inputs(case, seed)
    meshes = []
    for rest, tets, _, n, _, _ in bodies:
        dims = (n, 10 * n, n) if path == "batch" else (case["nx"], case["ny"], case["nz"])
        meshes.append(mg.TetMesh(rest, tets, dims))
    s = mg.Solver(meshes, _params(case))
    for b, ((_, _, fixed, _, E, nu), (x, v)) in enumerate(zip(bodies, states)):
        s.set_fixed(fixed, b)
        s.set_material(E, nu, b)
    if path == "diagnostics":
        s.set_state(*states[0])
        return {"path": path, "solver": s}
    net = None
    if case.get("learned"):
        net = MLP(device=0, seed=0)
        net.params = _trained_parameters()
        s.set_learned_smoother(net, 0.5)
    if case.get("split"):
        s.set_coarse_split(case["split"])
    if case.get("dense"):
        s.set_coarse_dense(True)
    if case.get("contact") == "triangles":
        s.set_surface_contact(True)
    for b, (x, v) in enumerate(states):
        s.set_state(x, v, b)
    a, e = tool - [half, 0, 0], tool + [half, 0, 0]
    return {"path": path, "solver": s, "net": net, "a": a.astype(np.float32), "b": e.astype(np.float32),
            "r": np.full(len(bodies), radius, np.float32), "frame": 0,
            **_frame_arrays(sum(len(m.positions) for m in meshes))}


def run(state):
    path, s = state["path"], state.get("solver")
    if path == "train":
        c, net = state["case"], state["net"]
        losses = net.train(state["x"], state["t"], steps=c["steps"], batch=c["batch"], lr=2e-3, seed=state["seed"])
        return {"losses": losses, "parameters": net.params}
    if path == "infer":
        return {"y": state["net"].forward(state["x"])}
    if path == "diagnostics":
        return {"normals": s.normals(), "energy": s.energy()}
    f = state["frame"] % TOOL_FRAMES
    state["frame"] += 1
    if path == "reference" and state["tool"] is not None:
        state["tool"].MoveTo(state["spheres"][f])
        s.Step()
        return {"positions": s.m_tetVertPos, "contact": s.m_tetVertIsCollide, "depth": s.m_tetVertCollisionDepth}
    if path == "reference":
        s.set_spheres(state["spheres"][f], [0.8])
        s.step()
        s.frame(state["positions"], state["contact"])
        return {"positions": state["positions"], "contact": state["contact"]}
    if path == "two_level":
        s.set_spheres(state["spheres"][f], [0.8])
        s.step()
        return {"fine": s.positions(0), "coarse": s.positions(1)}
    if len(state["r"]) == 1:
        s.set_capsule(state["a"][f, 0], state["b"][f, 0], float(state["r"][0]))
    else:
        s.set_capsules(state["a"][f], state["b"][f], state["r"])
    s.step()
    s.frame(state["positions"], state["contact"])
    return {"positions": state["positions"], "contact": state["contact"]}


def work(case):
    """State, tool, mesh and matrix read once, results written once; the arithmetic of the configured iterations."""
    path = case["path"]
    if path in ("train", "infer"):
        net = 2 * (9 * 64 + 64 * 64 + 64 * 3)
        if path == "infer":
            return {"bytes": 48 * case["rows"], "flops": net * case["rows"]}
        return {"bytes": 48 * case["pairs"] + 2 * 4 * 4995 + 4 * case["steps"],
                "flops": 3 * net * case["batch"] * case["steps"]}

    def box(n):
        return (n[0] + 1) * (n[1] + 1) * (n[2] + 1), 6 * n[0] * n[1] * n[2]

    if path == "batch":
        counts = [box((b[3], 10 * b[3], b[3])) for b in _batch(case)]
        V, T = sum(c[0] for c in counts), sum(c[1] for c in counts)
    elif case.get("shape") == "organ":
        rest, tets, _ = _body(case)
        V, T = len(rest), len(tets)
    else:
        V, T = box((case["nx"], case["ny"], case["nz"]))
    if path == "diagnostics":
        return {"bytes": 12 * V + 56 * T + 12 * V + 40, "flops": 400 * T}
    tet = 400   # F, its rotation and four corner forces
    if path in ("reference", "two_level"):
        if path == "two_level":
            cv, ct = box((case["cx"], case["cy"], case["cz"]))
            V, T = V + cv, T + ct
        return {"bytes": 56 * T + (24 + 4 + 28) * V, "flops": case["iterations"] * (tet * T + 60 * V)}
    passes, sweeps = case.get("passes", 1), case.get("sweeps", 2)
    nnz = 13 * V + 27 * V // 7    # level 0, and the coarse levels together
    smooth = 2 * (9 * 64 + 64 * 64 + 64 * 3) * V * 2 if case.get("learned") else 0
    cycle = 6 * nnz * (2 * sweeps + 1) + smooth + (12 * 13 * V if case.get("precision") == "mixed" else 0)
    return {"bytes": 56 * T + 8 * nnz + (24 + 28) * V, "flops": 10 * (tet * T + passes * cycle)}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(_device()).to(dtype)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _rotation(F):
    """Closest rotation of F [T, 3, 3]: Newton's iteration for the polar factor, the SVD where F turns a tet over."""
    X = F.clone()
    for _ in range(14):
        C = torch.stack([_cross(X[:, 1], X[:, 2]), _cross(X[:, 2], X[:, 0]), _cross(X[:, 0], X[:, 1])], 1)
        det = (X[:, 0] * C[:, 0]).sum(-1)
        g = ((C.square().sum((1, 2)) / X.square().sum((1, 2))).sqrt() / det.abs()).sqrt()
        X = 0.5 * (g[:, None, None] * X + C / (det * g)[:, None, None])
    bad = torch.nonzero(~(torch.linalg.det(F) > 0)).squeeze(1)
    if len(bad):
        U, S, Vh = torch.linalg.svd(F[bad].cpu())
        U[..., 2] *= torch.sign(torch.linalg.det(U) * torch.linalg.det(Vh))[:, None]
        X[bad] = (U @ Vh).to(X.device)
    return X


def _gradients(rest, tets):
    """Shape gradients g [T, 4, 3] and volumes of the rest tets."""
    p = rest[tets]
    D = torch.stack([p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], p[:, 3] - p[:, 0]], 2)
    inv = torch.linalg.inv(D)
    return torch.cat([-inv.sum(1, keepdim=True), inv], 1), torch.linalg.det(D).abs() / 6.0


def _deformation(x, tets, g):
    return torch.einsum("tji,tjk->tik", x[tets], g)


def _faces(tets):
    """Boundary faces [F, 3], wound outward for positively oriented tets."""
    f = torch.cat([tets[:, [0, 2, 1]], tets[:, [0, 1, 3]], tets[:, [0, 3, 2]], tets[:, [1, 2, 3]]])
    opposite = torch.cat([tets[:, 3], tets[:, 2], tets[:, 1], tets[:, 0]])
    s = f.sort(1).values
    n = int(tets.max()) + 1
    _, index, count = torch.unique((s[:, 0] * n + s[:, 1]) * n + s[:, 2], return_inverse=True, return_counts=True)
    once = count[index] == 1
    return f[once], opposite[once]


def _sparse(i, j, v, n, m):
    return torch.sparse_coo_tensor(torch.stack([i, j]), v, (n, m)).coalesce()


def _mul(A, x):
    return torch.sparse.mm(A, x)


class _Cycle:
    """The V-cycle's operators: Galerkin levels over voxel grids that halve their hexes, all bodies at once."""

    def __init__(self, rest, body, dims, A, fixed, levels, omega):
        self.omega, self.A, self.P = omega, [A], []
        nb = dims.shape[0]
        lo = torch.full((nb, 3), math.inf, dtype=rest.dtype, device=rest.device)
        hi = -lo
        lo = lo.scatter_reduce(0, body[:, None].expand(-1, 3), rest, "amin")
        hi = hi.scatter_reduce(0, body[:, None].expand(-1, 3), rest, "amax")
        pos, live = rest, ~fixed
        for _ in range(1, levels):
            dims = ((dims + 1) // 2).clamp(min=1)
            h = (hi - lo) / dims
            s = (pos - lo[body]) / h[body]
            cell = s.floor().to(torch.int64).clamp(min=0).minimum(dims[body] - 1)
            u = (s - cell).clamp(0.0, 1.0)
            val, perm = u.sort(dim=1, descending=True, stable=True)
            w = torch.stack([1 - val[:, 0], val[:, 0] - val[:, 1], val[:, 1] - val[:, 2], val[:, 2]], 1)
            w = torch.where(w < 1e-10, torch.zeros_like(w), w)
            w = w / w.sum(1, keepdim=True) * live[:, None]
            count = (dims + 1).prod(1)
            first = torch.cumsum(count, 0) - count
            key, at = [], cell.clone()
            for k in range(4):
                if k:
                    at = at.scatter_add(1, perm[:, k - 1:k], torch.ones_like(at[:, :1]))
                d = dims[body]
                key.append(first[body] + at[:, 0] + (d[:, 0] + 1) * (at[:, 2] + (d[:, 2] + 1) * at[:, 1]))
            key = torch.stack(key, 1)
            row = torch.arange(len(pos), device=pos.device)[:, None].expand(-1, 4)
            use = w > 0
            nodes, col = torch.unique(key[use], return_inverse=True)
            P = _sparse(row[use], col, w[use], len(pos), len(nodes))
            self.P.append(P)
            self.A.append(_mul(_mul(P.t().coalesce(), self.A[-1]), P).coalesce())
            body = torch.searchsorted(first + count, nodes, right=True)
            local = nodes - first[body]
            d = dims[body]
            grid = torch.stack([local % (d[:, 0] + 1), local // ((d[:, 0] + 1) * (d[:, 2] + 1)),
                                (local // (d[:, 0] + 1)) % (d[:, 2] + 1)], 1)
            pos = lo[body] + h[body] * grid
            live = torch.ones(len(nodes), dtype=torch.bool, device=pos.device)
        self.body, self.bodies = body, nb

    def contacts(self, c, fixed):
        """This frame's diagonals: the contact weights c lumped down, and the coarsest inverse."""
        self.D, self.off, self.inv = [], [], []
        for l, A in enumerate(self.A):
            i, v = A.indices(), A.values()
            on = i[0] == i[1]
            n = A.shape[0]
            D = torch.zeros(n, dtype=v.dtype, device=v.device).index_add(0, i[0][on], v[on]) + c
            self.D.append(D)
            self.off.append(_sparse(i[0][~on], i[1][~on], v[~on], n, n).to_sparse_csr())
            self.inv.append(torch.where(fixed, torch.zeros_like(D), self.omega / D) if l == 0 else self.omega / D)
            if l + 1 < len(self.A):
                c = _mul(self.P[l].t(), c[:, None])[:, 0]
        A, n = self.A[-1], self.A[-1].shape[0]
        size = torch.bincount(self.body, minlength=self.bodies)
        self.local = torch.arange(n, device=c.device) - (torch.cumsum(size, 0) - size)[self.body]
        dense = torch.eye(int(size.max()), dtype=c.dtype, device=c.device).repeat(self.bodies, 1, 1)
        i = A.indices()
        dense[self.body[i[0]], self.local[i[0]], self.local[i[1]]] = A.values()
        dense[self.body, self.local, self.local] = self.D[-1]
        self.coarsest = torch.linalg.inv(dense)

    def apply(self, l, x):
        return self.D[l][:, None] * x + _mul(self.off[l], x)

    def sweep(self, l, x, b):
        return x + self.inv[l][:, None] * (b - self.apply(l, x))

    def coarse(self, l, r, sweeps):
        """Correction of level l >= 1 for the right-hand side r."""
        if l + 1 == len(self.A):
            full = torch.zeros(self.bodies, self.coarsest.shape[1], 3, dtype=r.dtype, device=r.device)
            full[self.body, self.local] = r
            return (self.coarsest @ full)[self.body, self.local]
        e = torch.zeros_like(r)
        for _ in range(sweeps):
            e = self.sweep(l, e, r)
        e = e + _mul(self.P[l], self.coarse(l + 1, _mul(self.P[l].t(), r - self.apply(l, e)), sweeps))
        for _ in range(sweeps):
            e = self.sweep(l, e, r)
        return e


def _network(p, x):
    w1, b1, w2, b2, w3, b3 = (p[a:b] for a, b in ((0, 576), (576, 640), (640, 4736), (4736, 4800), (4800, 4992),
                                                  (4992, 4995)))
    h = torch.nn.functional.gelu(x @ w1.reshape(64, 9).T + b1, approximate="tanh")
    h = torch.nn.functional.gelu(h @ w2.reshape(64, 64).T + b2, approximate="tanh")
    return h @ w3.reshape(3, 64).T + b3


def _learned_sweep(cycle, p, diag, r, free):
    """scale * network(features) for the level-0 residual r (zero at fixed vertices)."""
    a = torch.sparse_csr_tensor(cycle.off[0].crow_indices(), cycle.off[0].col_indices(),
                                cycle.off[0].values().abs(), cycle.off[0].shape)
    D = cycle.D[0]
    sa = _mul(a, torch.ones_like(D)[:, None])[:, 0]
    ring, dring = _mul(a, r) / sa[:, None], _mul(a, D[:, None])[:, 0] / sa
    s = (r.square().sum(1) + ring.square().sum(1)).sqrt()
    safe = torch.where(s > 0, s, torch.ones_like(s))[:, None]
    x = torch.cat([r / safe, torch.stack([D / sa, (D - diag) / D, D / dring], 1), ring / safe], 1)
    return torch.where(free & (s > 0), s / D, torch.zeros_like(s))[:, None] * _network(p, x)


def _segment_triangle(a, b, c, p0, p1):
    """Closest points h on the triangles and q on the segment p0 p1, and where the segment passes through."""
    def clamp(t):
        return t.clamp(0.0, 1.0)

    def dot(u, v):
        return (u * v).sum(-1)

    best = torch.full(a.shape[:1], math.inf, dtype=a.dtype, device=a.device)
    h, q = a.clone(), p0.clone()

    def offer(hn, qn, ok=None):
        nonlocal best, h, q
        d = dot(hn - qn, hn - qn)
        d = d if ok is None else torch.where(ok, d, torch.full_like(d, math.inf))
        take = d < best
        best = torch.where(take, d, best)
        h, q = torch.where(take[:, None], hn, h), torch.where(take[:, None], qn, q)

    n = _cross(b - a, c - a)

    def inside(x):
        return ((dot(_cross(b - a, x - a), n) >= 0) & (dot(_cross(c - b, x - b), n) >= 0) &
                (dot(_cross(a - c, x - c), n) >= 0))

    for p in (p0, p1):                                    # an end of the segment over the face
        x = p - n * (dot(n, p - a) / dot(n, n))[:, None]
        offer(x, p, inside(x))
    d1 = p1 - p0
    for e0, e1 in ((a, b), (b, c), (c, a)):               # the segment and an edge, their ends included
        d2, r = e1 - e0, p0 - e0
        aa, ee, ff, cc, bb = dot(d1, d1), dot(d2, d2), dot(d2, r), dot(d1, r), dot(d1, d2)
        den = aa * ee - bb * bb
        s = torch.where(den > 0, clamp((bb * ff - cc * ee) / torch.where(den > 0, den, torch.ones_like(den))),
                        torch.zeros_like(den))
        t = (bb * s + ff) / ee
        s = torch.where(t < 0, clamp(-cc / aa), torch.where(t > 1, clamp((bb - cc) / aa), s))
        t = clamp(t)
        offer(e0 + d2 * t[:, None], p0 + d1 * s[:, None])
    s0, s1 = dot(n, p0 - a), dot(n, p1 - a)
    x = p0 + d1 * (s0 / torch.where(s0 == s1, torch.ones_like(s0), s0 - s1))[:, None]
    through = (s0 * s1 <= 0) & (s0 != s1) & inside(x)
    best = torch.where(through, torch.zeros_like(best), best)
    return h, q, best.sqrt(), n, through


def _capsule_contacts(case, s, body, faces, opposite, a, b, r):
    """Contact mask and targets on the predicted positions s, against each body's capsule."""
    surface = torch.zeros(len(s), dtype=torch.bool, device=s.device)
    surface[faces.reshape(-1)] = True
    A, B, R = a[body], b[body], r[body]
    ab = B - A
    t = (((s - A) * ab).sum(1) / ab.square().sum(1)).clamp(0.0, 1.0)
    q = A + t[:, None] * ab
    d = (s - q).square().sum(1).sqrt()
    hit = surface & (d < R)
    n = torch.where((d > 1e-12)[:, None], (s - q) / d.clamp(min=1e-300)[:, None],
                    torch.tensor([0.0, 0.0, 1.0], dtype=s.dtype, device=s.device))
    target = q + R[:, None] * n
    if case.get("contact") == "triangles":
        fb = body[faces[:, 0]]
        fa, fbv, fc = s[faces[:, 0]], s[faces[:, 1]], s[faces[:, 2]]
        h, qq, dist, nrm, _ = _segment_triangle(fa, fbv, fc, a[fb], b[fb])
        touch = (dist < r[fb]) & (r[fb] > 0)
        inward = nrm * torch.sign((nrm * (s[opposite] - fa)).sum(1))[:, None]
        inward = inward / inward.square().sum(1).sqrt()[:, None]
        push = torch.where((dist > 1e-12)[:, None], (h - qq) * ((r[fb] - dist) / dist.clamp(min=1e-300))[:, None],
                           inward * r[fb][:, None])
        total, many = torch.zeros_like(s), torch.zeros(len(s), dtype=s.dtype, device=s.device)
        for k in range(3):
            total = total.index_add(0, faces[touch][:, k], push[touch])
            many = many.index_add(0, faces[touch][:, k], torch.ones_like(push[touch][:, 0]))
        more = (many > 0) & ~hit
        target = torch.where(more[:, None], s + total / many.clamp(min=1.0)[:, None], target)
        hit = hit | more
    return hit, target


def _exact_frame(case, seed):
    bodies, states, tool, half, radius = _frame_inputs(case, seed)
    at = np.cumsum([0] + [len(b[0]) for b in bodies])
    rest = _t(np.concatenate([b[0] for b in bodies]))
    body = _t(np.repeat(np.arange(len(bodies)), np.diff(at)), torch.int64)
    tets = _t(np.concatenate([b[1].astype(np.int64) + o for b, o in zip(bodies, at)]), torch.int64)
    fixed = _t(np.concatenate([b[2] for b in bodies]), torch.bool)
    E = _t(np.concatenate([np.broadcast_to(b[4], len(b[1])) for b in bodies]))
    nu = _t(np.concatenate([np.broadcast_to(b[5], len(b[1])) for b in bodies]))
    x0 = _t(np.concatenate([s[0] for s in states]))
    v0 = _t(np.concatenate([s[1] for s in states]))
    n, one = len(rest), lambda f: float(np.float32(f))
    dt, damping, omega, kc = one(1.0 / 60.0), one(0.95), one(2.0 / 3.0), 1e6
    g, vol = _gradients(rest, tets)
    w = E / (1.0 + nu) * vol
    mass = torch.zeros(n, dtype=rest.dtype, device=rest.device)
    for k in range(4):
        mass = mass.index_add(0, tets[:, k], 1000.0 * vol / 4.0)
    gg = torch.einsum("tik,tjk->tij", g, g) * w[:, None, None]
    everyone = torch.arange(n, device=rest.device)
    A = _sparse(torch.cat([tets[:, :, None].expand(-1, 4, 4).reshape(-1), everyone]),
                torch.cat([tets[:, None, :].expand(-1, 4, 4).reshape(-1), everyone]),
                torch.cat([gg.reshape(-1), mass / (dt * dt)]), n, n)
    if case["path"] == "batch":
        dims = np.array([[b[3], 10 * b[3], b[3]] for b in bodies])
    else:
        dims = np.array([[case["nx"], case["ny"], case["nz"]]])
    cycle = _Cycle(rest, body, _t(dims, torch.int64), A, fixed, case["levels"], omega)
    free = (~fixed)[:, None].to(rest.dtype)
    gravity = torch.zeros(3, dtype=rest.dtype, device=rest.device)
    gravity[2 if case.get("shape") == "organ" else 1] = one(case.get("gravity", 0.0))
    v = (v0 * damping + gravity * dt) * free
    s = x0 + v * dt * free
    hit = torch.zeros(n, dtype=torch.bool, device=rest.device)
    target = s
    if radius > 0:
        faces, opposite = _faces(tets)
        a = _t((tool[0] - [half, 0, 0]).astype(np.float32))
        b = _t((tool[0] + [half, 0, 0]).astype(np.float32))
        hit, target = _capsule_contacts(case, s, body, faces, opposite, a, b,
                                        _t(np.full(len(bodies), radius, np.float32)))
    c = torch.where(hit & ~fixed, torch.full_like(mass, kc), torch.zeros_like(mass))
    cycle.contacts(c, fixed)
    diag = cycle.D[0] - c
    b0 = c[:, None] * (target - s)
    net = _t(_trained_parameters()) if case.get("learned") else None
    Fs = _deformation(s, tets, g)
    d = torch.zeros_like(s)
    sweeps = case.get("sweeps", 2)
    for _ in range(10):
        R = _rotation(_deformation(s + d, tets, g))
        force = torch.einsum("tik,tjk->tji", (R - Fs) * w[:, None, None], g)
        b = b0.index_add(0, tets.reshape(-1), force.reshape(-1, 3))
        for _ in range(case.get("passes", 1)):
            if net is not None:
                d = d + _learned_sweep(cycle, net, diag, free * (b - cycle.apply(0, d)), ~fixed)
            else:
                for _ in range(sweeps):
                    d = cycle.sweep(0, d, b)
            d = d + _mul(cycle.P[0], cycle.coarse(1, _mul(cycle.P[0].t(), b - cycle.apply(0, d)), sweeps))
            if net is not None:
                d = d + _learned_sweep(cycle, net, diag, free * (b - cycle.apply(0, d)), ~fixed)
            else:
                for _ in range(sweeps):
                    d = cycle.sweep(0, d, b)
    return {"positions": s + d, "contact": None}


class _Reference:
    """The reference's Jacobi/Chebyshev iteration on one mesh."""

    def __init__(self, rest, tets, fixed, x, v, drop):
        self.tets, self.drop = _t(tets, torch.int64), drop
        self.g, self.vol = _gradients(_t(rest), self.tets)
        self.free = 1.0 - _t(fixed)[:, None]
        n = len(rest)
        self.mass = torch.zeros(n, dtype=torch.float64, device=_device())
        self.diag = torch.zeros_like(self.mass)
        for k in range(4):
            self.mass = self.mass.index_add(0, self.tets[:, k], self.vol / 4.0)
            self.diag = self.diag.index_add(0, self.tets[:, k], self.g[:, k].square().sum(1) * self.vol * 8000.0)
        self.dt = float(np.float32(1.0 / 60.0))
        gravity = torch.tensor([0.0, float(np.float32(-9.8)), 0.0], dtype=torch.float64, device=_device())
        v = (_t(v) * float(np.float32(0.95)) + gravity * self.dt) * self.free
        self.s = _t(x) + v * self.dt * self.free
        self.x, self.last, self.omega = self.s, self.s, 1.0

    def forces(self):
        F = _deformation(self.x, self.tets, self.g)
        C = F.transpose(1, 2) @ F
        trace = C.diagonal(dim1=1, dim2=2).sum(1)
        spread = trace ** 2 - 1.5 * (trace ** 2 - (C @ C).diagonal(dim1=1, dim2=2).sum(1))
        # the reference takes a tet that is all but unstrained as a scaled rotation
        R = torch.where((spread < 1e-6)[:, None, None], F / (trace / 3.0).sqrt()[:, None, None], _rotation(F))
        f = torch.einsum("tik,tjk->tji", R - F, self.g).clamp(-10.0, 10.0)
        f = f * self.vol[:, None, None] * 8000.0
        if self.drop:
            f = torch.where(f.abs() < 1e-5, torch.zeros_like(f), f)
        return torch.zeros_like(self.x).index_add(0, self.tets.reshape(-1), f.reshape(-1, 3))

    def sphere(self, centre, r):
        """Diagonal and force of the vertices inside 1.5 radii, and how deep they are."""
        cp = self.x - centre
        dist = cp.square().sum(1).sqrt()
        u = cp / dist[:, None]
        inside = dist < 1.5 * r
        t = 1.5 * r - dist
        depth = torch.where(inside & (t > 0.5 * r), t - 0.5 * r, torch.zeros_like(t))
        on = inside.to(t.dtype)[:, None]
        return on * 1000.0 * u * u, on * 1000.0 * (t / 2.0)[:, None] * u, depth

    def iterate(self, cd, cf):
        rho = float(np.float32(0.9992))
        self.omega = 4.0 / (4.0 - rho * rho * self.omega)
        dc = (self.mass / self.dt ** 2)[:, None]
        step = (dc * (self.s - self.x) + self.forces() + cf) / (self.diag[:, None] + cd + dc) * self.free
        new = self.x + step * float(np.float32(0.6))
        new = self.omega * (new - self.last) + self.last
        self.last, self.x = self.x, new


def _exact_reference(case, seed):
    rest, tets, fixed, x, v = _reference_state(case, seed)
    if case["mirror"]:
        d = np.sqrt(((rest - np.array([0.0, 10.0, 0.0], np.float32)) ** 2).sum(1))
        fixed = (d < 1.8).astype(np.uint8)
    ref = _Reference(rest, tets, fixed, x, v, True)
    centre, r = _t(_sphere_path(case, seed)[0]), float(np.float32(0.8))
    depth = None
    for _ in range(case["iterations"]):
        cd, cf, depth = ref.sphere(centre, r)
        ref.iterate(cd, cf)
    if case["mirror"]:
        return {"positions": ref.x.reshape(-1), "contact": None, "depth": depth}
    return {"positions": ref.x, "contact": None}


def _sphere_triangles(x, faces, c, r):
    """Push c - hit and hit flag of each surface triangle against the sphere: face, outer edge cylinder, vertex."""
    def dot(u, v):
        return (u * v).sum(-1)

    V = [x[faces[:, k]] for k in range(3)]
    n = _cross(V[1] - V[0], V[2] - V[0])
    n = n / dot(n, n).sqrt()[:, None]
    sd = dot(n, c - V[0])
    near, proj = sd.abs() <= r, c - n * sd[:, None]
    v0, v1, v2 = V[2] - V[0], V[1] - V[0], proj - V[0]
    den = dot(v0, v0) * dot(v1, v1) - dot(v0, v1) ** 2
    p = (dot(v1, v1) * dot(v0, v2) - dot(v0, v1) * dot(v1, v2)) / den
    q = (dot(v0, v0) * dot(v1, v2) - dot(v0, v1) * dot(v0, v2)) / den
    found = (p >= 0) & (q >= 0) & (p + q <= 1)
    hit = c + n * ((r - sd.abs()) * torch.where(sd < 0, -torch.ones_like(sd), torch.ones_like(sd)))[:, None]
    for i in range(3):
        b, e, o = V[i], V[(i + 1) % 3], V[(i + 2) % 3]
        length = dot(e - b, e - b).sqrt()
        u = (e - b) / length[:, None]
        t = dot(c - b, u)
        on = b + u * t[:, None]
        rad = dot(c - on, c - on).sqrt()
        outer = dot(_cross(u, o - b), _cross(u, proj - b)) < 0
        ok = ~found & (t >= 0) & (t <= length) & (rad < r) & outer
        hit = torch.where(ok[:, None], on + (c - on) / rad[:, None] * r, hit)
        found = found | ok
    for i in range(3):
        dist = dot(c - V[i], c - V[i]).sqrt()
        ok = ~found & (dist <= r)
        hit = torch.where(ok[:, None], V[i] + (c - V[i]) / dist[:, None] * r, hit)
        found = found | ok
    found = (found & near).to(x.dtype)
    return (c - hit) * found[:, None], found


def _box_interpolation(points, nodes, nx, ny, nz):
    """Rows of barycentric weights of `points` in the Kuhn tets of a box mesh with nx, ny, nz hexes."""
    u = np.stack([(points[:, a].astype(np.float64) - lo) / (-2.0 * lo) * n
                  for a, (lo, n) in enumerate(((-1.0, nx), (-10.0, ny), (-1.0, nz)))], 1)
    cell = np.clip(np.floor(u + 1e-9).astype(int), 0, np.array([nx, ny, nz]) - 1)
    f = u - cell
    perm = np.argsort(-f, axis=1, kind="stable")
    val = np.take_along_axis(f, perm, 1)
    w = np.stack([1 - val[:, 0], val[:, 0] - val[:, 1], val[:, 1] - val[:, 2], val[:, 2]], 1)
    ids, at = [], cell.copy()
    for k in range(4):
        if k:
            at[np.arange(len(at)), perm[:, k - 1]] += 1
        ids.append(at[:, 0] + (nx + 1) * (at[:, 2] + (nz + 1) * at[:, 1]))
    return _t(np.stack(ids, 1), torch.int64), _t(w)


def _exact_two_level(case, seed):
    fine = _beam(case["nx"], case["ny"], case["nz"])
    coarse = _beam(case["cx"], case["cy"], case["cz"])
    C, F = (_Reference(m[0], m[1], m[2], m[0], np.zeros_like(m[0]), False) for m in (coarse, fine))
    faces, _ = _faces(C.tets)
    centre, r = _t(_sphere_path(case, seed)[0]), float(np.float32(0.8))
    for _ in range(case["iterations"]):
        push, count = _sphere_triangles(C.x, faces, centre, r)
        cf, cd = torch.zeros_like(C.x), torch.zeros_like(C.mass)
        for k in range(3):
            cf = cf.index_add(0, faces[:, k], 1000.0 * push)
            cd = cd.index_add(0, faces[:, k], 1000.0 * count)
        C.iterate(cd[:, None], cf)
    ids, w = _box_interpolation(fine[0], coarse[0], case["cx"], case["cy"], case["cz"])
    F.x = F.last = (C.x[ids] * w[:, :, None]).sum(1)
    for _ in range(case["iterations"]):
        cd, cf, _ = F.sphere(centre, r)
        F.iterate(cd, cf)
    ids, w = _box_interpolation(coarse[0], fine[0], case["nx"], case["ny"], case["nz"])
    return {"fine": F.x, "coarse": (F.x[ids] * w[:, :, None]).sum(1)}


def _exact_training(case, seed):
    x, t = _pairs(case["pairs"], seed)
    x, t = _t(x), _t(t)
    p = _t(_initial_parameters(seed)).requires_grad_()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    losses, steps, batch = [], case["steps"], case["batch"]
    with np.errstate(over="ignore"):
        for k in range(steps):
            z = (np.uint64(seed) + np.uint64(k) * np.uint64(0x9E3779B97F4A7C15)
                 + np.arange(batch, dtype=np.uint64) * np.uint64(0xBF58476D1CE4E5B9))
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            rows = _t(((z ^ (z >> np.uint64(31))) % np.uint64(case["pairs"])).astype(np.int64), torch.int64)
            loss = (_network(p, x[rows]) - t[rows]).square().mean()
            losses.append(loss.detach())
            (g,) = torch.autograd.grad(loss, p)
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            lr = 2e-3 * (0.55 + 0.45 * math.cos(math.pi * k / steps))
            with torch.no_grad():
                p -= lr * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"losses": torch.stack(losses), "parameters": p.detach()}


def _exact_diagnostics(case, seed):
    (body,), (state,), *_ = _frame_inputs(case, seed)
    rest, tets, x = _t(body[0]), _t(body[1], torch.int64), _t(state[0])
    faces, _ = _faces(tets)
    n = _cross(x[faces[:, 1]] - x[faces[:, 0]], x[faces[:, 2]] - x[faces[:, 0]])
    n = n / n.square().sum(1).sqrt()[:, None]
    normal = torch.zeros_like(x)
    for k in range(3):
        normal = normal.index_add(0, faces[:, k], n)
    length = normal.square().sum(1).sqrt()
    normal = torch.where((length > 0)[:, None], normal / length.clamp(min=1e-300)[:, None], normal)
    g, vol = _gradients(rest, tets)
    dt = float(np.float32(1.0 / 60.0))
    moved = (x - rest).square().sum(1)
    kinetic = sum((1000.0 * vol / 4.0 * moved[tets[:, k]]).sum() for k in range(4)) / (2.0 * dt * dt)
    F = _deformation(x, tets, g)
    w = _t(np.broadcast_to(body[4], len(body[1]))) / (1.0 + _t(body[5])) * vol
    elastic = (0.5 * w * (F - _rotation(F)).square().sum((1, 2))).sum()
    zero = torch.zeros_like(kinetic)
    return {"normals": normal, "energy": torch.stack([kinetic, elastic, zero, zero, zero])}


def exact(case, seed):
    path = case["path"]
    if path in ("frame", "batch"):
        return _exact_frame(case, seed)
    if path == "reference":
        return _exact_reference(case, seed)
    if path == "two_level":
        return _exact_two_level(case, seed)
    if path == "train":
        return _exact_training(case, seed)
    if path == "infer":
        return {"y": _network(_t(_trained_parameters()), _t(_pairs(case["rows"], seed)[0]))}
    return _exact_diagnostics(case, seed)
