"""The measured work of this framework: what its users have it do, through its
public entry points, over the sizes they do it at.

Frames (`kind` of a scene): a program holds a `GPUSolver`, submits `frames`
physics frames and reads the poses back; a vector environment also uploads new
motor targets before every frame and reads its motors afterwards.  The solver
goes on from pass to pass as a simulation does, from the contact regime that
`prepare` brings it to.  The other kinds are the warm-start network's training
step and inference, and the observation and render compute of a viewer or a
learner, which leave their results on the device.

The scenes come from the builders of `avbd_b200.demos` (the benchmark's own
configurations at the listed sizes); every seed starts from poses of its own.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "avbd-metal_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

from avbd_b200 import GPUSolver, abi, demos, learned, load_library  # noqa: E402

DIN, HID, DOUT, USED = learned.DIN, learned.HID, learned.DOUT, learned.USED


def listed():
    return [
        # an interactive program: one small scene, every frame read back
        {"name": "stack-20", "kind": "stack", "bodies": 20, "iterations": 10, "frames": 1, "preroll": 30},
        # a rigid scene just above the single-block solver, dynamic coloring
        {"name": "boxes-700", "kind": "boxes", "bodies": 700, "iterations": 10, "frames": 4, "preroll": 30},
        # a pile of capsules, tori, spheres, boxes and hulls
        {"name": "shapes-512", "kind": "shapes", "bodies": 512, "iterations": 10, "frames": 4, "preroll": 60},
        # a vector environment's step: targets in, one frame, motors and poses out
        {"name": "worlds-4096", "kind": "worlds", "worlds": 4096, "iterations": 8, "frames": 1, "preroll": 30},
        # one soft body, plain and with the learned warm start
        {"name": "soft-24", "kind": "soft", "n": 24, "iterations": 20, "frames": 4, "preroll": 40},
        {"name": "soft-24-learned", "kind": "soft-learned", "n": 24, "iterations": 10, "frames": 4, "preroll": 40},
        # cloth with self-contact (Planar-DAT)
        {"name": "cloth-256", "kind": "cloth", "n": 256, "iterations": 30, "frames": 4, "preroll": 60},
        # soft bodies, rigid boxes and cloth together (isotropic OGC)
        {"name": "mixed-64", "kind": "mixed", "cubes": 64, "cube_n": 10, "boxes": 256, "cloth_n": 128,
         "iterations": 20, "frames": 4, "preroll": 40},
        # the warm-start network: inference over a large batch, one Adam step at the trainer's batch
        {"name": "infer-1m", "kind": "infer", "rows": 1 << 20},
        {"name": "train-8192", "kind": "train", "rows": 8192},
        # pixel observations of a Push-T batch
        {"name": "obs-4096x64", "kind": "obs", "envs": 4096, "res": 64},
        # a viewer's smooth normals and skinned mesh of a soft body
        {"name": "render-24", "kind": "render", "n": 24, "per_tet": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stack", "boxes", "shapes", "worlds", "soft", "soft-learned", "cloth", "mixed", "infer",
                       "train", "obs", "render"])
    if kind == "stack":
        return {"kind": kind, "bodies": rng.randint(2, 24), "iterations": rng.randint(5, 20), "frames": 1,
                "preroll": rng.randint(20, 40)}
    if kind == "boxes":
        return {"kind": kind, "bodies": _log(rng, 60, 3000), "iterations": rng.randint(5, 16),
                "frames": rng.randint(1, 4), "preroll": rng.randint(20, 40)}
    if kind == "shapes":
        return {"kind": kind, "bodies": _log(rng, 40, 900), "iterations": rng.randint(5, 16),
                "frames": rng.randint(1, 4), "preroll": rng.randint(40, 70)}
    if kind == "worlds":
        return {"kind": kind, "worlds": _log(rng, 16, 4096), "iterations": rng.randint(4, 12), "frames": 1,
                "preroll": rng.randint(20, 40)}
    if kind in ("soft", "soft-learned"):
        return {"kind": kind, "n": rng.randint(6, 24), "iterations": rng.randint(8, 20),
                "frames": rng.randint(1, 4), "preroll": rng.randint(30, 50)}
    if kind == "cloth":
        return {"kind": kind, "n": _log(rng, 24, 256), "iterations": rng.randint(10, 30),
                "frames": rng.randint(1, 4), "preroll": rng.randint(40, 60)}
    if kind == "mixed":
        return {"kind": kind, "cubes": _log(rng, 4, 64), "cube_n": rng.randint(5, 10), "boxes": _log(rng, 16, 256),
                "cloth_n": rng.randint(32, 128), "iterations": rng.randint(8, 20), "frames": rng.randint(1, 4),
                "preroll": rng.randint(30, 50)}
    if kind == "infer":
        return {"kind": kind, "rows": _log(rng, 1, 1 << 20)}
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 200, 16384)}
    if kind == "obs":
        return {"kind": kind, "envs": _log(rng, 8, 4096), "res": rng.randint(32, 96)}
    return {"kind": kind, "n": rng.randint(6, 24), "per_tet": rng.randint(1, 4)}


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _scene(key):
    """(scene, motor joints or environments) of a case's sizes."""
    c = dict(key)
    kind = c["kind"]
    extra = None
    if kind == "stack":
        s = demos.rigid_stack_scene(count=c["bodies"])
    elif kind == "boxes":
        s = demos.box_field_scene(count=c["bodies"])
    elif kind == "shapes":
        s = demos.shapes_scene(count=c["bodies"])
    elif kind == "worlds":
        s, extra, _ = demos.batched_worlds_scene(worlds=c["worlds"])
    elif kind in ("soft", "soft-learned", "render"):
        s = demos.soft_cube_scene(n=c["n"], exclusion_joints=kind == "soft")
    elif kind == "cloth":
        s = demos.cloth_sphere_scene(n=c["n"])
    elif kind == "mixed":
        s = demos.mixed_scene(cubes=c["cubes"], cube_n=c["cube_n"], boxes=c["boxes"], cloth_n=c["cloth_n"])
    else:
        s, extra = demos.pusht_scene(num_envs=c["envs"])
    return s, extra


SIZES = ("kind", "bodies", "worlds", "n", "cubes", "cube_n", "boxes", "cloth_n", "envs")


def scene_of(case):
    s, extra = _scene(tuple((k, case[k]) for k in SIZES if k in case))
    if "iterations" in case:
        s.settings.iterations = case["iterations"]
    return s, extra


def start_positions(scene, seed, spread=1e-4):
    """The scene's body positions, every dynamic body moved by N(0, spread)."""
    rng = np.random.default_rng(seed)
    p = np.array([b.position for b in scene.bodies], np.float32)
    moves = np.array([b.is_dynamic for b in scene.bodies])
    return p + (rng.normal(0.0, spread, p.shape) * moves[:, None]).astype(np.float32)


class Frames:
    """A running simulation."""

    def __init__(self, case, seed):
        scene, self.motors = scene_of(case)
        self.solver = GPUSolver(scene)
        self.solver.set_positions(start_positions(scene, seed))
        self.frames = case["frames"]
        self.frame = 0
        if case["kind"] == "worlds":
            rng = np.random.default_rng(seed + 1)
            self.motors = np.array(self.motors, np.uint32)
            self.targets = rng.uniform(-0.5, 0.5, (16, len(self.motors))).astype(np.float32)
            for _ in range(case["preroll"]):
                self.drive()
                self.solver.step(1)
        else:
            self.motors = None
            self.solver.step(case["preroll"])
        if case["kind"] == "soft-learned":
            m = learned.WarmStartModel.load(os.path.join(PACKAGE, "avbd_b200", "models",
                                                         "soft_cube_24_warm_start.npz"))
            self.solver.set_warm_start_model(m.params, m.norm, 1, rigid=m.rigid)
            self.solver.set_warm_start_mode(abi.WARM_START_LEARNED)
            self.solver.step(4)
        self.solver.synchronize()

    def drive(self):
        self.solver.set_motor_targets(self.motors, self.targets[self.frame % len(self.targets)])
        self.frame += 1

    def run(self):
        g = self.solver
        if self.motors is None:
            g.step(self.frames)
            return g.positions()
        self.drive()
        g.step(1)
        return g.motor_states(self.motors) + g.positions()


# ---------------------------------------------------------------------------
# The warm-start network
# ---------------------------------------------------------------------------
def network(seed):
    """He-initialised parameters with small biases and a normalisation block, in float32."""
    rng = np.random.default_rng(seed)
    parts = []
    for out, inp, scale in ((HID, DIN, 1.0), (HID, HID, 1.0), (HID, HID, 1.0), (DOUT, HID, 0.5)):
        parts += [rng.normal(0.0, scale * math.sqrt(2.0 / inp), out * inp), rng.normal(0.0, 0.05, out)]
    prm = np.concatenate(parts).astype(np.float32)
    norm = np.concatenate([rng.normal(0.0, 0.5, DIN), rng.uniform(0.5, 2.0, DIN), rng.normal(0.0, 0.1, DOUT),
                           rng.uniform(0.5, 2.0, DOUT)]).astype(np.float32)
    return torch.from_numpy(prm).cuda(), torch.from_numpy(norm).cuda()


def batch(rows, seed, norm):
    """Features spread as the normalisation expects, and targets that depend on them."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn(rows, DIN, device="cuda", generator=gen) / norm[DIN:2 * DIN] + norm[:DIN]
    mix = torch.randn(DIN, USED, device="cuda", generator=gen) / math.sqrt(DIN)
    t = torch.tanh(((x - norm[:DIN]) * norm[DIN:2 * DIN]) @ mix) + 0.1 * torch.randn(rows, USED, device="cuda",
                                                                                     generator=gen)
    return x.contiguous(), (t * norm[80:80 + USED] + norm[64:64 + USED]).contiguous()


def check(rc):
    if rc != 0:
        raise RuntimeError(f"status {rc}")


class Infer:
    def __init__(self, case, seed):
        self.lib = load_library()
        self.prm, self.norm = network(seed)
        self.x, _ = batch(case["rows"], seed + 1, self.norm)
        self.out = torch.zeros(case["rows"], USED, device="cuda")
        self.ws = torch.empty(1 << 17, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        check(self.lib.avbd_mlp_infer(self.prm.data_ptr(), self.norm.data_ptr(), self.x.data_ptr(), len(self.x),
                                      self.out.data_ptr(), self.ws.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream))
        return self.out


FIRST_STEP, LR = 200, 1e-3


class Train:
    """A training run in its 200th step: Adam moments of a gradient's size."""

    def __init__(self, case, seed):
        self.lib = load_library()
        self.prm, self.norm = network(seed)
        self.x, self.t = batch(case["rows"], seed + 1, self.norm)
        self.m, self.v = moments(self.prm, seed)
        self.step = FIRST_STEP
        self.ws = torch.zeros(self.lib.avbd_mlp_workspace_bytes(case["rows"]), dtype=torch.uint8, device="cuda")
        self.loss = torch.zeros(1, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        check(self.lib.avbd_mlp_train_step(self.prm.data_ptr(), self.norm.data_ptr(), self.x.data_ptr(),
                                           self.t.data_ptr(), len(self.x), self.m.data_ptr(), self.v.data_ptr(),
                                           self.step, ctypes.c_float(LR), self.ws.data_ptr(), self.loss.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream))
        self.step += 1
        return {"params": self.prm, "m": self.m, "v": self.v, "loss": self.loss}


def moments(prm, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 2)
    m = 1e-3 * torch.randn(prm.shape, device="cuda", generator=gen)
    v = 1e-4 * (0.1 + torch.rand(prm.shape, device="cuda", generator=gen))
    return m, v


# ---------------------------------------------------------------------------
# Observations and render compute
# ---------------------------------------------------------------------------
class Obs:
    def __init__(self, case, seed):
        scene, envs = scene_of(case)
        self.solver = GPUSolver(scene)
        self.solver.set_positions(start_positions(scene, seed, 0.1))
        self.table = demos.pusht_env_table(envs)
        self.res = case["res"]
        self.out = torch.zeros(case["envs"], self.res, self.res, 3, dtype=torch.uint8, device="cuda")
        self.solver.synchronize()
        torch.cuda.synchronize()

    def run(self):
        self.solver.render_pusht_obs(self.table, self.res, device_out=self.out.data_ptr())
        return self.out


@functools.lru_cache(maxsize=2)
def _bindings(n, per_tet):
    scene, _ = scene_of({"kind": "render", "n": n})
    b = demos.skin_bindings_for_tets(scene, per_tet)
    return (abi.SkinBinding * len(b))(*b)


class Render:
    def __init__(self, case, seed):
        scene, _ = scene_of(case)
        self.solver = GPUSolver(scene)
        self.solver.set_skin_bindings(_bindings(case["n"], case["per_tet"]))
        self.solver.set_positions(deformed(scene, case, seed))
        self.normals = torch.zeros(len(scene.bodies), 4, device="cuda")
        self.skin = torch.zeros(len(scene.tets) * case["per_tet"], 8, device="cuda")
        self.solver.synchronize()
        torch.cuda.synchronize()

    def run(self):
        self.solver.soft_normals(device_out=self.normals.data_ptr())
        self.solver.skin_deform(device_out=self.skin.data_ptr())
        return {"normals": self.normals, "skin": self.skin}


def deformed(scene, case, seed):
    """A smooth bend of the rest lattice and a little noise, float32."""
    p = start_positions(scene, seed, 0.02 / (case["n"] - 1))
    w = np.random.default_rng(seed + 1).uniform(-0.1, 0.1, (3, 3)).astype(np.float32)
    d = np.array([b.is_dynamic for b in scene.bodies])
    p[d] += np.sin(2.0 * p[d]).astype(np.float32) @ w
    return p.astype(np.float32)


# ---------------------------------------------------------------------------
MAKERS = {"infer": Infer, "train": Train, "obs": Obs, "render": Render}


def prepare(case, seed):
    return MAKERS.get(case["kind"], Frames)(case, seed)


def run(state):
    return state.run()


#: Floating-point operations of one visit of a constraint in one iteration
#: (stamp and dual), and of one body's solve, to the nearest hundred or so.
STAMP = {"tet": 600, "tri": 400, "spring": 100, "joint": 800, "contact": 400, "body": 200}


def work(case):
    kind = case["kind"]
    if kind in ("infer", "train"):
        n, weights = case["rows"], DIN * HID + 2 * HID * HID + HID * DOUT
        params = weights + 3 * HID + DOUT
        if kind == "infer":
            return {"bytes": 4 * n * (DIN + USED) + 4 * params, "flops": 2 * n * weights}
        # forward, weight gradients, and input gradients of all but the first layer
        return {"bytes": 4 * n * (DIN + USED) + 4 * 6 * params, "flops": 2 * n * (3 * weights - DIN * HID)}
    if kind == "obs":
        return {"bytes": case["envs"] * (3 * case["res"] ** 2 + 48 + 3 * 32), "flops": 0}
    if kind == "render":
        n = case["n"]
        tets, surface = 5 * (n - 1) ** 3, 6 * n * n
        return {"bytes": 16 * n ** 3 + 2 * 16 * surface + 16 * 2 * surface + case["per_tet"] * tets * (96 + 32),
                "flops": case["per_tet"] * tets * 100 + 2 * surface * 150}
    # frames: every record of the scene read once, its poses and multipliers
    # written once; the sweeps visit every constraint in every iteration
    bodies = tets = tris = springs = joints = contacts = 0
    if kind == "stack":
        bodies, contacts = case["bodies"], 4 * case["bodies"]
    elif kind == "boxes":
        bodies, contacts = case["bodies"], 4 * case["bodies"]
    elif kind == "shapes":
        bodies, contacts = case["bodies"], 4 * case["bodies"]
    elif kind == "worlds":
        bodies, joints, contacts = 7 * case["worlds"], 6 * case["worlds"], 28 * case["worlds"]
    elif kind in ("soft", "soft-learned"):
        bodies, tets, contacts = case["n"] ** 3, 5 * (case["n"] - 1) ** 3, case["n"] ** 2
    elif kind == "cloth":
        bodies, tris, springs = case["n"] ** 2, 2 * (case["n"] - 1) ** 2, 2 * case["n"] ** 2
    else:
        soft, sheet = case["cubes"] * case["cube_n"] ** 3, case["cloth_n"] ** 2
        bodies, tets = soft + sheet + case["boxes"], 5 * case["cubes"] * (case["cube_n"] - 1) ** 3
        tris, springs, contacts = 2 * sheet, 2 * sheet, case["cubes"] * case["cube_n"] ** 2 + 4 * case["boxes"]
    sweep = (STAMP["tet"] * 4 * tets + STAMP["tri"] * 3 * tris + STAMP["spring"] * 3 * springs
             + STAMP["joint"] * 3 * joints + STAMP["contact"] * 3 * contacts + STAMP["body"] * bodies)
    record = 64 * tets + 48 * tris + 64 * springs + 224 * joints + 80 * contacts + 160 * bodies
    state = 80 * bodies + 96 * joints + 80 * contacts + 16 * springs
    return {"bytes": case["frames"] * (record + state), "flops": case["frames"] * case["iterations"] * sweep}


# ---------------------------------------------------------------------------
# In 64 bits
# ---------------------------------------------------------------------------
def _layers(prm):
    out, at = [], 0
    for o, i in ((HID, DIN), (HID, HID), (HID, HID), (DOUT, HID)):
        w = prm[at:at + o * i].reshape(o, i)
        at += o * i
        out.append((w, prm[at:at + o]))
        at += o
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "infer":
        prm, norm = (v.double() for v in network(seed))
        x, _ = batch(case["rows"], seed + 1, norm.float())
        h = (x.double() - norm[:DIN]) * norm[DIN:2 * DIN]
        layers = _layers(prm)
        for w, b in layers[:3]:
            h = torch.relu(h @ w.T + b)
        w, b = layers[3]
        y = (h @ w.T + b)[:, :USED]
        return y * norm[80:80 + USED] + norm[64:64 + USED]
    if kind == "train":
        prm32, norm32 = network(seed)
        x, t = batch(case["rows"], seed + 1, norm32)
        m, v = (q.double() for q in moments(prm32, seed))
        prm, norm = prm32.double().requires_grad_(True), norm32.double()
        h = (x.double() - norm[:DIN]) * norm[DIN:2 * DIN]
        layers = _layers(prm)
        for w, b in layers[:3]:
            h = torch.relu(h @ w.T + b)
        w, b = layers[3]
        y = (h @ w.T + b)[:, :USED]
        tn = (t.double() - norm[64:64 + USED]) / norm[80:80 + USED]
        loss = ((y - tn) ** 2).sum() / case["rows"]
        loss.backward()
        g = prm.grad
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        mh, vh = m / (1.0 - 0.9 ** FIRST_STEP), v / (1.0 - 0.999 ** FIRST_STEP)
        p = prm.detach() - LR * mh / (vh.sqrt() + 1e-8)
        return {"params": p, "m": m, "v": v, "loss": loss.detach().reshape(1)}
    if kind == "render":
        return _exact_render(case, seed)
    return None  # an iterative solver's frames; observations are bytes


def _unit(v):
    return v / np.maximum(np.linalg.norm(v, axis=-1, keepdims=True), 1e-300)


def _exact_render(case, seed):
    scene, _ = scene_of(case)
    rest = np.array([b.position for b in scene.bodies], np.float32).astype(np.float64)
    p = deformed(scene, case, seed).astype(np.float64)
    tets = np.array([t.ids for t in scene.tets])
    # the boundary faces, turned outwards by the vertex opposite to them
    faces = np.concatenate([tets[:, [1, 2, 3]], tets[:, [0, 2, 3]], tets[:, [0, 1, 3]], tets[:, [0, 1, 2]]])
    inner = np.concatenate([tets[:, 0], tets[:, 1], tets[:, 2], tets[:, 3]])
    _, index, count = np.unique(np.sort(faces, axis=1), axis=0, return_index=True, return_counts=True)
    faces, inner = faces[index[count == 1]], inner[index[count == 1]]
    a, b, c = (rest[faces[:, k]] for k in range(3))
    inwards = np.einsum("ij,ij->i", np.cross(b - a, c - a), rest[inner] - a) > 0
    faces[inwards] = faces[inwards][:, [0, 2, 1]]
    a, b, c = (p[faces[:, k]] for k in range(3))
    fn = np.cross(b - a, c - a)
    area = 0.5 * np.linalg.norm(fn, axis=1)
    acc, wsum = np.zeros_like(p), np.zeros(len(p))
    for at, u, v in ((0, b - a, c - a), (1, a - b, c - b), (2, a - c, b - c)):
        w = area * np.arccos(np.clip(np.einsum("ij,ij->i", _unit(u), _unit(v)), -1.0, 1.0))
        np.add.at(acc, faces[:, at], _unit(fn) * w[:, None])
        np.add.at(wsum, faces[:, at], w)
    on = np.unique(faces)
    normals = np.zeros((len(p), 4))
    normals[on, :3] = _unit(acc[on])
    radius = np.array([b.size[0] for b in scene.bodies], np.float64)[on] * 0.5
    coherence = np.clip((np.linalg.norm(acc[on], axis=1) / wsum[on]) ** 2, 0.0, 1.0)
    normals[on, 3] = np.abs(radius) * (0.25 + 0.75 * coherence)
    bind = np.frombuffer(_bindings(case["n"], case["per_tet"]),
                         dtype=[("ids", "u4", 4), ("w", "f4", 4), ("n", "f4", 4), ("inv", "f4", (3, 4))])
    q = p[bind["ids"].astype(np.int64)]
    pos = np.einsum("ij,ijk->ik", bind["w"].astype(np.float64), q)
    r = rest[bind["ids"].astype(np.int64)]
    ds, dm = (np.stack([v[:, k] - v[:, 0] for k in (1, 2, 3)], axis=2) for v in (q, r))
    f = ds @ np.linalg.inv(dm)
    n0 = _unit(bind["n"][:, :3].astype(np.float64))
    cof = np.stack([np.cross(f[:, :, 1], f[:, :, 2]), np.cross(f[:, :, 2], f[:, :, 0]),
                    np.cross(f[:, :, 0], f[:, :, 1])], axis=2)
    skin = np.zeros((len(bind), 8))
    skin[:, :3], skin[:, 3] = pos, 1.0
    skin[:, 4:7] = _unit(np.einsum("ijk,ik->ij", cof, n0))
    return {"normals": normals, "skin": skin}
