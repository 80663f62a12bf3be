"""Performance cases of the contact solver: what its users run, through the
package's public entry points, over the range of sizes they run it at.

  solve  one scene from host arrays (lib.Solver.solve): the call a simulation
         makes once per step in place of ForceSolver::fillForces;
  batch  many independent scenes in one call, packed in device memory
         (lib.Solver.batch_solve_device) or in page-locked host memory
         (lib.Solver.batch_solve);
  world  one step of a device-resident world (lib.World: contact detection,
         solve and integration), from host state and back to it;
  mesh   the contacts of every neighbouring pair of mesh bodies
         (lib.mesh_contacts_pairs).

The contact problems are settled ones (residual velocities ~ 2 mm/s), which the solver's interior-point
iteration determines far below 1e-9: stacks and piles of boxes with 4 corner
contacts per touching face pair at the default tolerance (1e-6, 100
iterations); crates of cubes packed face to face, columns of tilted contacts,
worlds and pits at a scene file's (1e-4, 50).  Scenes in violent motion end at
the iteration cap at a point that depends on the last bit of every sum (two
correct executions differ by up to 1e-2 there), so they are not among them.
"""
import math

import numpy as np
import torch

from primal_dual_contacts_miror_b200 import abi, lib, scenes

GRAVITY = (0.0, 0.0, -9.81)
DT = 0.01
MU = 0.5
REST = 0.002
MESH_ROWS = 128  # output rows per mesh pair
DEFAULT = {"tol": 1e-6, "iters": 100}  # the solver's defaults
FILE = {"tol": 1e-4, "iters": 50}      # a scene file's settings


def listed():
    return [
        # the single-scene workload: a 10-box stack, one solve per step, where
        # the latency of the call is what counts
        {"name": "solve_stack_10", "kind": "solve", "scene": "stack", "n": 10, **DEFAULT},
        # one dense scene of an interactive simulation: a crate of 144 cubes,
        # whose contact graph is a 3-D grid (fill-in, a long elimination tree)
        {"name": "solve_crate_144", "kind": "solve", "scene": "crate", "nx": 6, "ny": 6, "nz": 4, **FILE},
        # the batched workload: 4,096 scenes of 4 to 256 bodies, device arrays
        {"name": "batch_piles_4096", "kind": "batch", "scene": "pile", "scenes": 4096, "lo": 4, "hi": 256,
         "host": False, "normal": False, "spring": False, **DEFAULT},
        # batched scenes with dense contact graphs, as heaps and crates have
        {"name": "batch_crates_1024", "kind": "batch", "scene": "crate", "scenes": 1024, "lo": 1, "hi": 6,
         "host": False, "normal": False, "spring": False, **FILE},
        # a rollout that keeps its state in host memory, with a friction
        # coefficient per contact
        {"name": "batch_columns_host_256", "kind": "batch", "scene": "columns", "scenes": 256, "lo": 2, "hi": 32,
         "host": True, "normal": False, "spring": False, **FILE},
        # thousands of the smallest scenes, frictionless force model
        {"name": "batch_normal_2048", "kind": "batch", "scene": "pile", "scenes": 2048, "lo": 1, "hi": 24,
         "host": False, "normal": True, "spring": False, **DEFAULT},
        # large single scenes: sparse direct solve of a loose pile, a packed
        # crate whose factor is too deep (conjugate gradients to 1e-13), and
        # above 2,000 bodies the iterative branch
        {"name": "large_pile_1900", "kind": "solve", "scene": "pile", "n": 1900, **DEFAULT},
        {"name": "large_crate_1152", "kind": "solve", "scene": "crate", "nx": 12, "ny": 12, "nz": 8, **FILE},
        {"name": "large_pile_6000", "kind": "solve", "scene": "pile", "n": 6000, **DEFAULT},
        # a step of 1,024 worlds of 4 to 256 boxes, columns at rest on the
        # ground and boxes still falling above them
        {"name": "world_boxes_1024", "kind": "world", "scene": "boxes", "scenes": 1024, "lo": 4, "hi": 256, **FILE},
        # a step of one pit of 50,000 spheres: sort-based contact detection and
        # the iterative branch on the whole GPU
        {"name": "world_pit_50000", "kind": "world", "scene": "pit", "scenes": 1, "lo": 50000, "hi": 50000, **FILE},
        # a chain of 32 mesh links, every neighbouring pair in one call
        {"name": "mesh_chain_32", "kind": "mesh", "links": 32, "around": 38, "tube": 15},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "large", "batch", "batch", "batch", "world", "mesh"])
    if kind == "solve":
        if rng.random() < 0.5:
            return {"kind": "solve", "scene": "stack", "n": _log_int(rng, 1, 40), **DEFAULT}
        return {"kind": "solve", "scene": "crate", "nx": rng.randint(1, 6), "ny": rng.randint(1, 6),
                "nz": rng.randint(1, 6), **FILE}
    if kind == "large":
        if rng.random() < 0.6:
            return {"kind": "solve", "scene": "pile", "n": _log_int(rng, 150, 6000), **DEFAULT}
        return {"kind": "solve", "scene": "crate", "nx": rng.randint(5, 12), "ny": rng.randint(5, 12),
                "nz": rng.randint(4, 8), **FILE}
    if kind == "batch":
        scene = rng.choice(["pile", "pile", "crate", "columns"])
        host, model = rng.random() < 0.4, rng.random()
        most = {"pile": 4096, "crate": 1024, "columns": 256}[scene]
        hi = {"pile": _log_int(rng, 8, 256), "crate": rng.randint(2, 6), "columns": _log_int(rng, 8, 32)}[scene]
        return {"kind": "batch", "scene": scene, "scenes": _log_int(rng, 8, most), "lo": 1, "hi": hi, "host": host,
                "normal": scene != "columns" and model < 0.2, "spring": scene == "pile" and model > 0.85,
                **(DEFAULT if scene == "pile" else FILE)}
    if kind == "world":
        if rng.random() < 0.7:
            return {"kind": "world", "scene": "boxes", "scenes": _log_int(rng, 1, 1024), "lo": 4,
                    "hi": _log_int(rng, 8, 256), **FILE}
        n = _log_int(rng, 2500, 50000)
        return {"kind": "world", "scene": "pit", "scenes": 1, "lo": n, "hi": n, **FILE}
    return {"kind": "mesh", "links": _log_int(rng, 2, 32), "around": rng.randint(12, 38), "tube": rng.randint(8, 15)}


# ------------------------------------------------------------------- inputs
def _columns(n, rng):
    """Columns of 1 to 4 large boxes, n in all, contact normals tilted by ~0.02
    rad and a friction coefficient per contact: the package's settled pile with
    those two drawn anew."""
    s = scenes.settled_pile(n, rng, max_height=4, half_range=(0.25, 0.75), vel_noise=REST)
    nrm = np.concatenate([rng.normal(0.0, 0.02, (s.n_contacts, 2)), np.ones((s.n_contacts, 1))], 1)
    s.frame = _frames(nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).reshape(-1, 9)
    s.mu = rng.uniform(0.3, 0.8, s.n_contacts)
    return s


def _frames(n):
    """Rotations taking the x axis onto the normals n: columns n, t1, t2."""
    ax = np.stack([np.zeros(len(n)), -n[:, 2], n[:, 1]], 1)
    an = np.sqrt((ax * ax).sum(1))
    ang = np.arctan2(an, n[:, 0])
    ax = ax / np.where(an > 0, an, 1.0)[:, None]
    c, s = np.cos(ang), np.sin(ang)
    k = np.zeros((len(n), 3, 3))
    k[:, 0, 1], k[:, 0, 2], k[:, 1, 2] = -ax[:, 2], ax[:, 1], -ax[:, 0]
    k -= k.transpose(0, 2, 1)
    return c[:, None, None] * np.eye(3) + s[:, None, None] * k + (1 - c)[:, None, None] * ax[:, :, None] * ax[:, None]


def _contact_scenes(case, seed):
    rng, sizes = np.random.default_rng(seed), _sizes(case)
    if case["kind"] == "solve":
        if case["scene"] == "stack":
            return [scenes.resting_box_stack(case["n"], vel_noise=REST, rng=rng)]
        if case["scene"] == "crate":
            return [scenes.packed_lattice(case["nx"], case["ny"], case["nz"], rng, vel_noise=REST)]
        return [scenes.settled_pile(case["n"], rng, vel_noise=REST)]
    out = []
    for size in sizes:
        if case["scene"] == "crate":
            out.append(scenes.packed_lattice(*size, rng, vel_noise=REST))
        else:
            out.append(_columns(size, rng) if case["scene"] == "columns" else scenes.settled_pile(size, rng, vel_noise=REST))
    return out


def _sizes(case):
    """Bodies of each scene of a batch or a world, log-uniform in [lo, hi] (a
    crate: its three sides, uniform); they belong to the case, not to the seed."""
    if "scenes" not in case:
        return []
    rng = np.random.default_rng([case["scenes"], case["lo"], case["hi"]])
    if case["scene"] == "crate":
        return [tuple(int(k) for k in rng.integers(case["lo"], case["hi"] + 1, 3)) for _ in range(case["scenes"])]
    return [int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(case["scenes"])]


def _config(case):
    return abi.default_config(tol=case["tol"], max_iter=case["iters"], mu=MU, spring_based=int(case.get("spring", False)),
                              force_model=int(case.get("normal", False)))


def _box_world(n, rng):
    """Half of the boxes in columns of 1 to 4 at rest (0.1 mm of overlap, random
    yaw, velocities ~ 2 mm/s) on a walled floor, the others in the air above,
    at random orientations and falling."""
    side = max(1.0, 0.6 * math.ceil(math.sqrt(n / 4.0)))
    half = rng.uniform(0.05, 0.2, (n, 3))
    rest = n - n // 2
    pos, quat = np.zeros((n, 3)), np.zeros((n, 4))
    col, k = 0, 0
    cells = max(1, int(side / 0.6))
    while k < rest:
        z = 0.0
        for k in range(k, min(rest, k + int(rng.integers(1, 5)))):
            pos[k] = (0.3 + 0.6 * (col % cells), 0.3 + 0.6 * (col // cells), z + half[k, 2] - 1e-4)
            z = pos[k, 2] + half[k, 2]
            yaw = rng.uniform(-0.3, 0.3)
            quat[k] = (0.0, 0.0, math.sin(yaw / 2), math.cos(yaw / 2))
        col, k = col + 1, k + 1
    width = 0.6 * (col // cells + 1)
    fall = np.arange(rest, n)
    pos[fall] = np.stack([rng.uniform(0.4, max(0.41, side - 0.4), len(fall)),
                          rng.uniform(0.4, max(0.41, width - 0.4), len(fall)), 4.0 + 0.75 * np.arange(len(fall))], 1)
    q = rng.normal(size=(len(fall), 4))
    quat[fall] = q / np.linalg.norm(q, axis=1, keepdims=True)
    vel, ang = rng.normal(0, REST, (n, 3)), rng.normal(0, REST, (n, 3))
    vel[fall, 2] -= rng.uniform(0, 10, len(fall))
    mass = 1000.0 * 8.0 * half.prod(1)
    sq = half * half
    inertia = mass[:, None] / 3.0 * np.stack([sq[:, 1] + sq[:, 2], sq[:, 0] + sq[:, 2], sq[:, 0] + sq[:, 1]], 1)
    return _walled(0, half, pos, quat, vel, ang, mass, inertia, max(side, 0.6 * cells), width)


def _pit_world(n, rng):
    """n spheres of radius 0.02 to 0.05 m in layers on a jittered lattice over
    the ground, about one contact per two spheres, as a filling pit has."""
    r = rng.uniform(0.04, 0.05, n)
    d = 0.097
    side = max(1, int(round(n ** (1 / 3) * 1.1)))
    k = np.arange(n)
    i, j, l = k % side, (k // side) % side, k // (side * side)
    pos = np.stack([i * d + (l % 2) * d / 2, j * d + (l % 2) * d / 2, l * d * math.sqrt(0.5)], 1)
    pos += rng.normal(0.0, 0.02 * d, (n, 3))
    pos -= pos.min(0)
    pos += (0.06, 0.06, 0.0392)
    mass = 1000.0 * 4.0 / 3.0 * math.pi * r ** 3
    quat = np.tile((0.0, 0.0, 0.0, 1.0), (n, 1))
    size = np.stack([r, 0 * r, 0 * r], 1)
    inertia = np.repeat((0.4 * mass * r * r)[:, None], 3, 1)
    return _walled(1, size, pos, quat, rng.normal(0, REST, (n, 3)), rng.normal(0, REST, (n, 3)), mass, inertia,
                   d * (side + 2), d * (side + 2))


def _walled(kind, size, pos, quat, vel, ang, mass, inertia, lx, ly):
    """Shape arrays with the ground and four walls (planes) in front."""
    s = math.sqrt(0.5)
    planes = [((0, 0, 0), (0, 0, 0, 1)), ((0, 0, 0), (0, s, 0, s)), ((lx, 0, 0), (0, -s, 0, s)),
              ((0, 0, 0), (-s, 0, 0, s)), ((0, ly, 0), (s, 0, 0, s))]
    n, p = len(mass), len(planes)
    pad = lambda a, fill: np.concatenate([np.full((p,) + a.shape[1:], fill), a])
    out = {"type": np.r_[np.full(p, 2), np.full(n, kind)], "size": pad(size, 0.0), "pos": pad(pos, 0.0),
           "quat": pad(quat, 0.0), "vel": pad(vel, 0.0), "ang_vel": pad(ang, 0.0), "mass": pad(mass, 1.0),
           "inertia0": pad(inertia, 1.0), "is_static": np.r_[np.ones(p, int), np.zeros(n, int)]}
    for q, (x, o) in enumerate(planes):
        out["pos"][q], out["quat"][q] = x, o
    return out


def _world_shapes(case, seed):
    rng = np.random.default_rng(seed)
    if case["scene"] == "pit":
        return [_pit_world(case["lo"], rng)]
    return [_box_world(n, rng) for n in _sizes(case)]


def _link_mesh(around, tube, major=0.5, minor=0.1):
    a = np.arange(around)[:, None] * (2 * math.pi / around)
    t = np.arange(tube)[None, :] * (2 * math.pi / tube)
    verts = np.stack([(major + minor * np.cos(t)) * np.cos(a), (major + minor * np.cos(t)) * np.sin(a),
                      minor * np.sin(t) + 0 * a], -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(around), np.arange(tube), indexing="ij")
    p = lambda x, y: ((x % around) * tube + y % tube).ravel()
    tris = np.concatenate([np.stack([p(i, j), p(i + 1, j), p(i + 1, j + 1)], 1),
                           np.stack([p(i, j), p(i + 1, j + 1), p(i, j + 1)], 1)])
    return verts, tris


def _chain(case, seed):
    """Link meshes (a little different each) and poses: every second link
    turned a quarter about the chain, neighbours 1 cm into each other."""
    rng = np.random.default_rng(seed)
    verts, tris = _link_mesh(case["around"], case["tube"])
    shapes = [verts * (1.0 + rng.uniform(-0.004, 0.004, 3)) for _ in range(case["links"])]
    poses = np.zeros((case["links"], 7))
    for k in range(case["links"]):
        q = np.r_[math.sin(math.pi / 4 * (k % 2)), 0.0, 0.0, math.cos(math.pi / 4 * (k % 2))] + rng.normal(0, 0.02, 4)
        poses[k] = np.r_[0.812 * k, rng.normal(0, 0.004, 2), q / np.linalg.norm(q)]
    return shapes, tris, poses


def prepare(case, seed):
    if case["kind"] == "mesh":
        shapes, tris, poses = _chain(case, seed)
        meshes = [lib.Mesh(v, tris) for v in shapes]
        pairs = [(meshes[k], poses[k], meshes[k + 1], poses[k + 1]) for k in range(case["links"] - 1)]
        return {"kind": "mesh", "pairs": pairs, "out": lib.mesh_contact_buffers(MESH_ROWS * len(pairs))}
    if case["kind"] == "world":
        shapes = abi.ShapeBatch(_world_shapes(case, seed), DT, GRAVITY)
        state = [lib.pinned_copy(a) for a in (shapes.pos, shapes.quat, shapes.vel, shapes.ang_vel)]
        return {"kind": "world", "world": lib.World(shapes, cfg=_config(case)), "state": state,
                "out": [lib.pinned_copy(a) for a in state], "stats": (abi.Stats * shapes.n_scenes)()}
    sc = _contact_scenes(case, seed)
    solver = lib.Solver(_config(case))
    if case["kind"] == "solve":
        return {"kind": "solve", "solver": solver, "scene": sc[0]}
    batch = abi.HostBatch(sc, DT, GRAVITY)
    if case["host"]:
        out = tuple(lib.pinned_copy(a) for a in abi.result_arrays(batch.all.n_bodies, batch.all.n_contacts))
        return {"kind": "host", "solver": solver, "batch": lib.pin_batch(batch), "out": out}
    return {"kind": "device", "solver": solver, "batch": lib.DeviceBatch(batch)}


def run(state):
    """Velocity increments and contact impulses (solve, batch), the bodies'
    state after the step (world), contact points (mesh: the rows the call
    writes, the others stay zero).  The solver's diagnostics (residuals at
    exit, trial counts) are no outputs of the path."""
    kind = state["kind"]
    if kind == "solve":
        return state["solver"].solve(state["scene"], dt=DT, gravity=GRAVITY)[:3]
    if kind == "host":
        return state["solver"].batch_solve(state["batch"], out=state["out"])[:3]
    if kind == "device":
        dev = state["batch"]
        state["solver"].batch_solve_device(dev, torch.cuda.current_stream().cuda_stream)
        return dev.out_dvel, dev.out_dang, dev.out_lf
    if kind == "world":
        world, stream = state["world"], torch.cuda.current_stream().cuda_stream
        world.set_state(*state["state"], stream=stream)
        world.step(1, stream=stream)
        world.get_state_async(*state["out"], stats=state["stats"], stream=stream)
        world.sync()  # a program reads its state here
        return state["out"]
    return {**state["out"], "counts": lib.mesh_contacts_pairs(state["pairs"], out=state["out"])["counts"]}


def work(case):
    """Bytes: every input array read once, every output written once.  Flops:
    one Newton iteration's contact terms and body blocks, contact detection not
    counted; for meshes the separating-axis tests of the neighbouring pairs'
    triangles that overlap (about a hundredth of them) and the distances of
    their vertices."""
    if case["kind"] == "mesh":
        tris, pairs = 2 * case["around"] * case["tube"], case["links"] - 1
        verts = tris // 2
        return {"bytes": 8 * case["links"] * (3 * verts + 1.5 * tris) + 200.0 * pairs * verts / 40,
                "flops": pairs * (tris * 60.0 + verts / 20 * tris * 60.0)}
    if case["kind"] == "world":
        n = case["scenes"] * _mean_size(case)
        return {"bytes": n * (2 * 13 * 8 + 11 * 8), "flops": n * 2000.0}
    if case["kind"] == "solve":
        n = case["n"] if "n" in case else case["nx"] * case["ny"] * case["nz"]
        nc = 4.0 * n if "n" in case else 4.0 * (3 * n - case["ny"] * case["nz"] - case["nx"] * case["nz"])
    elif case["scene"] == "crate":
        side = (case["lo"] + case["hi"]) / 2
        n = case["scenes"] * side ** 3
        nc = 4.0 * (3 * n - 2 * case["scenes"] * side ** 2)
    else:
        n = case["scenes"] * _mean_size(case)
        nc = 4.0 * n
    return {"bytes": n * (19 * 8 + 1 + 6 * 8) + nc * (2 * 4 + 16 * 8 + 3 * 8), "flops": nc * 600.0 + n * 1500.0}


def _mean_size(case):
    lo, hi = case["lo"], case["hi"]
    return lo if lo == hi else (hi - lo) / math.log(hi / lo)


# ------------------------------------------------------- values in 64 bits
def exact(case, seed):
    """The same Newton iteration, and the same contact rule, in plain numpy.
    None where that takes minutes: worlds, and batches and single scenes of
    thousands of bodies (dense factors here)."""
    if case["kind"] == "mesh":
        pairs = (case["links"] - 1) * (2 * case["around"] * case["tube"]) ** 2
        return _exact_mesh(*_chain(case, seed)) if pairs < 6e7 else None
    if case["kind"] == "world":
        return None
    if case["kind"] == "solve":
        n = case["n"] if "n" in case else case["nx"] * case["ny"] * case["nz"]
        return _newton(_contact_scenes(case, seed)[0], case) if n <= 300 else None
    if case["scenes"] > 100 or (case["scene"] == "crate" and case["scenes"] > 64) or (
            case["scene"] == "pile" and case["scenes"] * case["hi"] > 8000):
        return None
    got = [_newton(s, case) for s in _contact_scenes(case, seed)]
    return tuple(np.concatenate([g[k] for g in got]) for k in range(3))


def _cone(f, mu):
    """Friction cone sqrt(ft^2 + p) - mu fn - sqrt(p) - shift."""
    return np.sqrt(f[:, 1] ** 2 + f[:, 2] ** 2 + 1e-16) - mu * f[:, 0] - 1e-8 - 1e-8


def _radius(fn, mu):
    k = mu * fn + 1e-8 + 1e-8
    return np.sqrt(k * k - 1e-16)


def _sym(p):
    return np.stack([p[:, 0], p[:, 3], p[:, 4], p[:, 3], p[:, 1], p[:, 5], p[:, 4], p[:, 5], p[:, 2]],
                    1).reshape(-1, 3, 3)


def _newton(s, case):
    nb, nc = s.n_bodies, s.n_contacts
    g = np.array(GRAVITY)
    dvel, dang = np.tile(g * DT, (nb, 1)), np.zeros((nb, 3))
    if nc == 0:
        return dvel, dang, np.zeros((0, 3))
    static, mu = s.is_static != 0, (np.full(nc, MU) if s.mu is None else s.mu)
    normal, spring = case.get("normal", False), case.get("spring", False)
    body, R, arm = s.body, s.frame.reshape(-1, 3, 3), s.arm.reshape(-1, 2, 3)
    local = np.zeros(nb, bool)
    local[body] = True
    act = np.nonzero(local & ~static)[0]
    na, col = len(act), np.full(nb, -1)
    col[act] = np.arange(na)
    J, Ji = _sym(s.inertia), _sym(s.inv_inertia)

    def rel(u):  # R^T [(v1 + w1 x c1) - (v0 + w0 x c0)]
        p = [u[body[:, j], :3] + np.cross(u[body[:, j], 3:], arm[:, j]) for j in (0, 1)]
        return np.einsum("nji,nj->ni", R, p[1] - p[0])

    def scatter(x):  # sum over a body's contacts of sigma [x; c x x]
        out = np.zeros((nb, 6))
        for j, sg in ((0, -1.0), (1, 1.0)):
            np.add.at(out, body[:, j], sg * np.concatenate([x, np.cross(arm[:, j], x)], 1))
        out[static] = 0.0
        return out

    # characteristic mass and speed
    ve = np.concatenate([s.vel + np.where(static[:, None], 0.0, g * DT), s.ang_vel], 1)
    half = [np.einsum("nji,nj->ni", R, ve[body[:, j], :3] + np.cross(ve[body[:, j], 3:], arm[:, j])) for j in (0, 1)]
    nrel = np.linalg.norm(half[1] - half[0], axis=1)
    spd = np.zeros(nb)
    has_static = static[body[:, 0]] | static[body[:, 1]]
    for j in (0, 1):
        h = np.linalg.norm(half[j], axis=1)
        np.maximum.at(spd, body[:, j], np.where(has_static, np.maximum(h, nrel), h))
    cm = (3 * s.mass[act] + J[act].trace(axis1=1, axis2=2)).sum() / na / 6 if na else 1.0
    cs = max((spd[act] * s.mass[act]).sum() / s.mass[act].sum() if na else 0.0, np.linalg.norm(g) * DT * 0.25, 1e-4)
    u = np.concatenate([s.vel, s.ang_vel], 1) / cs
    uold = ve / cs
    n_loc = int(local.sum())
    tk = DT * 1e6
    compliance, reduction = 1.0 / (DT * (tk + 0.01 * 1e6)), tk / (tk + 0.01 * 1e6)
    extra = compliance * cm if spring else 0.0
    k_n = -reduction * s.depth / DT / cs if spring else 0.0 * s.depth
    q = np.zeros((nc, 2, 2))
    for j in (0, 1):
        a = np.cross(arm[:, j, :, None], R[:, :, 1:], axis=1)
        move = ~static[body[:, j]]
        m = np.einsum("nia,nib->nab", R[:, :, 1:], R[:, :, 1:]) / s.mass[body[:, j], None, None]
        q += np.where(move[:, None, None], m + np.einsum("nia,nij,njb->nab", a, Ji[body[:, j]], a), 0.0)
    f = np.tile([1.0, 0.0, 0.0], (nc, 1))
    lam = np.tile([1e-2, 0.0 if normal else 1e-2], (nc, 1))
    n_u, n_f, n_c = 6 * n_loc, (1 if normal else 3) * nc, (1 if normal else 2) * nc
    mass = np.zeros((nb, 6, 6))
    mass[:, range(3), range(3)] = s.mass[:, None] / cm
    mass[:, 3:, 3:] = J / cm

    def grad(f):
        if normal:
            return np.zeros((nc, 2))
        return f[:, 1:] / np.sqrt(f[:, 1] ** 2 + f[:, 2] ** 2 + 1e-16)[:, None]

    def cons(f):
        return np.stack([-f[:, 0], np.zeros(nc) if normal else _cone(f, mu)], 1)

    def residual(uv, w, f, lam):
        r = -w.copy()
        if normal:
            r[:, 1:] = 0.0
        if spring:
            r[:, 0] -= compliance * cm * f[:, 0]
        r[:, 0] += lam[:, 0] - k_n
        if not normal:
            r[:, 1:] -= lam[:, 1:] * grad(f)
        tn = np.linalg.norm(w[:, 1:], axis=1)
        th = w[:, 1:] / np.where(tn > 0, tn, 1.0)[:, None]
        rad = _radius(f[:, 0], mu)
        wt = np.minimum(rad / (tn + 1e-8) * np.einsum("na,nab,nb->n", th, q, th) * cm, 1.0)
        wr = r * np.stack([np.ones(nc), wt, wt], 1)
        a0 = np.maximum(f[:, 0] - (w[:, 0] + k_n + extra * f[:, 0]), 0.0) - f[:, 0]
        ac2 = a0 @ a0
        if not normal:
            td = f[:, 1:] - w[:, 1:]
            tdn = np.linalg.norm(td, axis=1)
            out = ~(tdn < rad)
            td = td * np.where(out, rad / np.where(out, tdn, 1.0), 1.0)[:, None]
            ac2 += ((td - f[:, 1:]) ** 2).sum()
        ff = f * np.array([1.0, 0.0, 0.0]) if normal else f
        ru = np.einsum("nij,nj->ni", mass, uv - uold) + scatter(-np.einsum("nij,nj->ni", R, ff))
        ru[static | ~local] = 0.0
        return r, (wr * wr).sum(), ac2, ru, (ru * ru).sum()

    hu = 1e-4
    for _ in range(case["iters"]):
        w = rel(u)
        c, gr = cons(f), grad(f)
        rf, wrf2, ac2, ru, ru2 = residual(u, w, f, lam)
        gap = -(lam * c).sum() / n_c
        muc = 0.1 * gap
        rl = lam * c + muc
        if normal:
            rl[:, 1] = 0.0
        rl2 = (rl * rl).sum()
        err, sac = ru2 + wrf2 + rl2, ru2 + ac2 + rl2
        eps = hu * err ** (0.66667 * 0.5)
        mom = math.sqrt(ru2) / n_u
        exit_err = max(mom, math.sqrt(wrf2) / n_f, math.sqrt(rl2) / n_c, gap)
        if min(exit_err, max(mom, math.sqrt(ac2) / nc)) < case["tol"]:
            break
        ic = np.stack([1.0 / (c[:, 0] - eps * (1.0 if normal else lam[:, 0])),
                       np.zeros(nc) if normal else 1.0 / (c[:, 1] - eps * lam[:, 1])], 1)
        sf = rf.copy()
        sf[:, 0] -= rl[:, 0] * ic[:, 0]
        sf[:, 1:] += gr * (rl[:, 1] * ic[:, 1])[:, None]
        kinv = np.zeros((nc, 3, 3))
        kinv[:, 0, 0] = 1.0 / (eps - lam[:, 0] * ic[:, 0] + (compliance * cm if spring else 0.0))
        if not normal:
            z = np.stack([f[:, 2], -f[:, 1]], 1)
            r3 = (f[:, 1] ** 2 + f[:, 2] ** 2 + 1e-6) ** -1.5
            hess = (z[:, :, None] * z[:, None] + 1e-6 * np.eye(2)) * r3[:, None, None]
            kt = eps * np.eye(2) - (lam[:, 1] * ic[:, 1])[:, None, None] * gr[:, :, None] * gr[:, None]
            kinv[:, 1:, 1:] = np.linalg.inv(kt + lam[:, 1][:, None, None] * hess)
        rhs = scatter(np.einsum("nij,njk,nk->ni", R, kinv, sf)) - ru
        W = np.einsum("nij,njk,nlk->nil", R, kinv, R)
        A = np.zeros((na, 6, na, 6))
        A[np.arange(na), :, np.arange(na)] = mass[act] + eps * np.eye(6)
        T = [np.concatenate([np.tile(np.eye(3), (nc, 1, 1)), np.cross(arm[:, j, :, None], np.eye(3)[None], axis=1)], 1)
             for j in (0, 1)]
        for a in (0, 1):
            for b in (0, 1):
                both = ~static[body[:, a]] & ~static[body[:, b]]
                blk = (1.0 if a == b else -1.0) * np.einsum("nij,njk,nlk->nil", T[a], W, T[b])
                np.add.at(A.transpose(0, 2, 1, 3), (col[body[both, a]], col[body[both, b]]), blk[both])
        du = np.zeros((nb, 6))
        if na:
            du[act] = np.linalg.solve(A.reshape(6 * na, 6 * na), rhs[act].reshape(-1)).reshape(-1, 6)
        wd = rel(du)
        df = np.einsum("nij,nj->ni", kinv, sf - wd)
        dl = np.stack([-ic[:, 0] * (-lam[:, 0] * df[:, 0] + rl[:, 0]),
                       -ic[:, 1] * (lam[:, 1] * (gr * df[:, 1:]).sum(1) + rl[:, 1])], 1)

        def search(du, wd, df, dl, most):
            step = 1.0
            for t in range(most):
                ft = f + step * df
                cut = ft[:, 0] < 0
                ft[cut, 0] = 0.0
                out = _cone(ft, mu) > 0
                tn = np.linalg.norm(ft[:, 1:], axis=1)
                ft[out, 1:] *= (np.maximum(_radius(ft[:, 0], mu), 0.0)[out] / tn[out])[:, None]
                d = np.where((cut | out)[:, None], ft - f, step * df)
                e = step * dl
                e = np.where((e < 0) & (lam + e < 0), -lam, e)
                fi, li, ui = f + 0.99 * d, lam + 0.99 * e, u + 0.99 * step * du
                r, wr2, a2, rb, rb2 = residual(ui, w + 0.99 * step * wd, fi, li)
                cl = li * cons(fi) + muc
                if normal:
                    cl[:, 1] = 0.0
                l2 = (cl * cl).sum()
                k = 1 if normal else 2
                slope = -(step * du * rb).sum() + (d * r).sum() + (e[:, :k] / li[:, :k] * cl[:, :k]).sum()
                ok = rb2 + wr2 + l2 < err or rb2 + a2 + l2 < sac
                if (ok and slope > 0) or t == most - 1:
                    return (step, ui, fi, li) if ok else (0.0, u, f, lam)
                step *= 0.5
            return 0.0, u, f, lam

        step, un, fn, ln = search(du, wd, df, dl, 10)
        full = step == 1.0
        if step == 0.0:
            full = False
            _, un, fn, ln = search(-ru, -rel(ru), rf, rl, 20)
        u, f, lam = un, fn, ln
        hu = max(hu / 4 if full else hu * 4, 1e-6)
    dvel[local], dang[local] = u[local, :3] * cs - s.vel[local], u[local, 3:] * cs - s.ang_vel[local]
    return dvel, dang, f * cs * cm


def _rot(q):
    x, y, z, w = q
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                     [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                     [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])


def _unit(v):
    n = np.linalg.norm(v, axis=-1, keepdims=True)
    return v / np.where(n > 0, n, 1.0)


def _exact_mesh(shapes, tris, poses):
    models = [_normals(v, tris) for v in shapes]
    rows, counts = [], []
    for k in range(len(poses) - 1):
        got = _mesh_pair(models[k], poses[k], models[k + 1], poses[k + 1], tris)
        counts.append(len(got[2]))
        rows.append(got)
    out = {}
    for i, key in enumerate(("pos", "normal", "depth", "frame", "arm")):
        got = np.concatenate([r[i] for r in rows])[: MESH_ROWS * len(rows)]
        out[key] = np.zeros((MESH_ROWS * len(rows),) + got.shape[1:])
        out[key][: len(got)] = got
    out["counts"] = np.array(counts, np.int32)
    return out


def _normals(v, tris):
    a, b, c = (v[tris[:, k]] for k in range(3))
    face = _unit(np.cross(b - a, c - a))
    vert, edge = np.zeros_like(v), {}
    for k in range(3):
        e1, e2 = (_unit(v[tris[:, (k + j) % 3]] - v[tris[:, k]]) for j in (1, 2))
        np.add.at(vert, tris[:, k], np.arccos(np.clip((e1 * e2).sum(1), -1, 1))[:, None] * face)
        for t, key in enumerate(np.sort(tris[:, [(k + 1) % 3, (k + 2) % 3]], 1).tolist()):
            edge[tuple(key)] = edge.get(tuple(key), 0.0) + face[t]
    return v, face, _unit(vert), edge


def _mesh_pair(ma, pa, mb, pb, tris):
    Ra, Rb = _rot(pa[3:]), _rot(pb[3:])
    wa, wb = ma[0] @ Ra.T + pa[:3], mb[0] @ Rb.T + pb[:3]
    P, Q = wa[tris], wb[tris]
    over = np.ones((len(tris), len(tris)), bool)
    for r in range(3):
        over &= P[:, :, r].min(1)[:, None] <= Q[:, :, r].max(1)[None]
        over &= Q[:, :, r].min(1)[None] <= P[:, :, r].max(1)[:, None]
    i, j = np.nonzero(over)
    p, q = P[i], Q[j]
    ep, eq = np.roll(p, -1, 1) - p, np.roll(q, -1, 1) - q
    n1, n2 = np.cross(ep[:, 0], -ep[:, 2]), np.cross(eq[:, 0], -eq[:, 2])
    axes = [n1, n2] + [np.cross(ep[:, x], eq[:, y]) for x in range(3) for y in range(3)]
    axes += [np.cross(n1, ep[:, x]) for x in range(3)] + [np.cross(n2, eq[:, x]) for x in range(3)]
    apart = np.zeros(len(i), bool)
    for L in axes:
        x, y = np.einsum("nij,nj->ni", p, L), np.einsum("nij,nj->ni", q, L)
        apart |= ((L * L).sum(1) >= 1e-30) & ((x.max(1) < y.min(1)) | (y.max(1) < x.min(1)))
    seeds = np.unique(tris[i[~apart]]), np.unique(tris[j[~apart]])
    pts = []
    for seed, w, m, R, c, sign in ((seeds[0], wa, mb, Rb, pb[:3], -1.0), (seeds[1], wb, ma, Ra, pa[:3], 1.0)):
        for v in seed:
            d, n = _signed(m, tris, (w[v] - c) @ R)
            if d < 0:
                pts.append((w[v], sign * (R @ n), -d))
    pos = np.array([x[0] for x in pts]).reshape(-1, 3)
    nrm = np.array([x[1] for x in pts]).reshape(-1, 3)
    dep = np.array([x[2] for x in pts])
    key = np.rint(pos * 1e9)
    o = np.lexsort((key[:, 2], key[:, 1], key[:, 0]))
    pos, nrm, dep = pos[o], nrm[o], dep[o]
    first = np.r_[True, ((pos[1:] - pos[:-1]) ** 2).sum(1) > 1e-8][: len(pos)]
    start = np.nonzero(first)[0]
    if len(start):
        many = np.diff(np.r_[start, len(pos)]) > 1
        total, least = np.add.reduceat(nrm, start), np.minimum.reduceat(dep, start)
        nrm = np.where(many[:, None], _unit(total), nrm[start])
        pos, dep = pos[start], least
    return pos, nrm, np.abs(dep), _frames(nrm).reshape(-1, 9), np.concatenate([pos - pa[:3], pos - pb[:3]], 1)


def _signed(m, tris, p):
    """Signed distance of p to the closed mesh m (first of the closest
    triangles, sign by its pseudonormal) and the vertex normals interpolated at
    the closest point."""
    v, face, vert, edge = m
    a, b, c = (v[tris[:, k]] for k in range(3))
    ab, ac, bc = b - a, c - a, c - b
    dot = lambda x, y: (x * y).sum(-1)
    d1, d2, d3, d4, d5, d6 = dot(ab, p - a), dot(ac, p - a), dot(ab, p - b), dot(ac, p - b), dot(ab, p - c), dot(ac, p - c)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    with np.errstate(all="ignore"):
        den = 1.0 / (va + vb + vc)
        bary = np.stack([1 - vb * den - vc * den, vb * den, vc * den], 1)
        t = (d4 - d3) / ((d4 - d3) + (d5 - d6))
        on = lambda *x: np.stack([np.broadcast_to(y, va.shape) for y in x], 1)
        for test, value in (((va <= 0) & (d4 >= d3) & (d5 >= d6), on(0.0, 1 - t, t)),
                            ((vb <= 0) & (d2 >= 0) & (d6 <= 0), on(1 - d2 / (d2 - d6), 0.0, d2 / (d2 - d6))),
                            ((d6 >= 0) & (d5 <= d6), on(0.0, 0.0, 1.0)),
                            ((vc <= 0) & (d1 >= 0) & (d3 <= 0), on(1 - d1 / (d1 - d3), d1 / (d1 - d3), 0.0)),
                            ((d3 >= 0) & (d4 <= d3), on(0.0, 1.0, 0.0)),
                            ((d1 <= 0) & (d2 <= 0), on(1.0, 0.0, 0.0))):
            bary = np.where(test[:, None], value, bary)
    q = bary[:, :1] * a + bary[:, 1:2] * b + bary[:, 2:] * c
    d2_ = dot(p - q, p - q)
    t = int(np.argmin(d2_))
    small = bary[t] <= 1e-12
    if small.sum() == 2:
        pn = vert[tris[t, int(np.argmin(small))]]
    elif small.sum() == 1:
        k = int(np.argmax(small))
        pn = _unit(edge[tuple(sorted((tris[t, (k + 1) % 3], tris[t, (k + 2) % 3])))])
    else:
        pn = face[t]
    dist = math.sqrt(d2_[t]) * (1.0 if dot(p - q[t], pn) >= 0 else -1.0)
    return dist, _unit(bary[t] @ vert[tris[t]])
