"""What a user of the framework has it do: rollouts of worlds, gradients through them, and candidate pairs.

A rollout is what a program that plans, trains or replays does with a batch: put a saved state back, then for each
frame add the frame's forces, step, and read every body's pose to the host. Putting the state back also makes
every pass the same work, however often it runs. Launch shapes are the library's own defaults. The scenes are
twofold_b200.scenes' (the repository's benchmark configurations and test worlds, over a range of sizes), each made
from the seed.

Outputs are the last poses of every body (rollouts), the final state and every gradient (adjoint), the keys and
their count (candidates). The library computes a rollout in float with the reference's operations in the
reference's order, branches on every comparison of it, and amplifies a changed bit from contact to contact; a
64-bit run is another trajectory, and the contact set an adjoint walks is one of such a run. So there is no value
in 64 bits to compare with: exact() has none.
"""
import ctypes as C
import math

import numpy as np
import torch

from twofold_b200 import abi, scenes
from twofold_b200.world import Batch

DT = float(np.float32(1.0 / 60.0))


def listed():
    return [
        # A game's frame loop on a handful of boxes, through the plain step the C++ World calls: launches and waits.
        {"name": "boxes_8", "kind": "boxes", "size": 8, "warm": 40, "frames": 4, "per_call": 1, "graph": False, "forces": False},
        # The box pyramid of the benchmark: one world of 210 bodies, a long chain of contacts.
        {"name": "pyramid_210", "kind": "pyramid", "size": 20, "warm": 24, "frames": 4, "per_call": 1, "graph": True, "forces": False},
        # One world of hulls, boxes and spheres: general polyhedra, where collision dominates; plain steps.
        {"name": "hulls_96", "kind": "hulls", "size": 96, "warm": 48, "frames": 4, "per_call": 1, "graph": False, "forces": False},
        # The large mixed scene of the benchmark: spheres, boxes and hulls falling on a terrain mesh.
        {"name": "terrain_32768", "kind": "terrain", "size": 32768, "warm": 36, "frames": 2, "per_call": 1, "graph": True, "forces": False},
        # The planar pile of the benchmark: the 2D path, contacts solved one at a time by level, mixed pairs.
        {"name": "planar_16384", "kind": "planar", "size": 16384, "warm": 30, "frames": 2, "per_call": 1, "graph": True, "forces": False},
        # A small batch of uneven worlds, one control per frame.
        {"name": "uneven_64", "kind": "uneven", "size": 64, "warm": 16, "frames": 4, "per_call": 1, "graph": True, "forces": True},
        # The headline workload: 4096 uneven worlds, forces in and poses out every frame.
        {"name": "uneven_4096", "kind": "uneven", "size": 4096, "warm": 16, "frames": 4, "per_call": 1, "graph": True, "forces": True},
        # Walls of boxes hit by a sphere: every world is refreshed mid-step; a control held over two steps.
        {"name": "impact_1024", "kind": "impact", "size": 1024, "warm": 16, "frames": 2, "per_call": 2, "graph": True, "forces": True},
        # A batch of jointed worlds (chains, doors, motors, springs), as articulated bodies are trained.
        {"name": "jointed_256", "kind": "jointed", "size": 256, "warm": 16, "frames": 4, "per_call": 1, "graph": True, "forces": True},
        # The model forward and the adjoint backward of the differentiable impact, in float.
        {"name": "adjoint_256_f32", "kind": "adjoint", "size": 256, "warm": 0, "frames": 48, "precision": 32},
        # The same in double, as gradients are checked.
        {"name": "adjoint_24_f64", "kind": "adjoint", "size": 24, "warm": 0, "frames": 24, "precision": 64},
        # Candidate pairs from device arrays inside another framework's frame.
        {"name": "candidates_4096", "kind": "candidates", "size": 4096},
    ]


# kind: (smallest, largest size, frames, warm-up steps, share of the draws)
RANGES = {
    "boxes": (1, 64, 4, (10, 60), 2),
    "pyramid": (2, 32, 4, (4, 40), 2),
    "hulls": (4, 160, 4, (20, 60), 1),
    "prisms": (4, 160, 4, (20, 60), 1),
    "cylinders": (4, 120, 4, (20, 60), 1),
    "bullets": (6, 96, 4, (0, 12), 1),
    "terrain": (256, 32768, 2, (24, 44), 2),
    "planar": (256, 16384, 2, (16, 60), 2),
    "uneven": (2, 4096, 4, (6, 24), 4),
    "impact": (4, 1024, 2, (6, 24), 2),
    "jointed": (1, 256, 4, (4, 30), 2),
    "adjoint": (2, 256, 0, (0, 0), 2),
    "candidates": (2, 4096, 0, (0, 0), 1),
}


def _log_size(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choices(list(RANGES), weights=[r[4] for r in RANGES.values()])[0]
    low, high, frames, warm, _ = RANGES[kind]
    size = _log_size(rng, low, high)
    if kind == "candidates":
        return {"kind": kind, "size": size}
    if kind == "adjoint":
        precision = rng.choice([32, 32, 64])
        return {"kind": kind, "size": size if precision == 32 else max(2, size // 10), "warm": 0,
                "frames": rng.randint(4, 48 if precision == 32 else 24), "precision": precision}
    per_call = rng.choice([1, 1, 2])
    return {"kind": kind, "size": size, "warm": rng.randint(*warm), "frames": max(1, frames // per_call),
            "per_call": per_call, "graph": rng.random() < 0.7, "forces": rng.random() < 0.5}


def _scene(case, seed):
    kind, n = case["kind"], case["size"]
    if kind == "boxes":
        return scenes.Scene(kind, [scenes.single("boxes", n=n, seed=seed)])
    if kind == "pyramid":
        return scenes.Scene(kind, [scenes.pyramid(n, seed=seed)])
    if kind in ("hulls", "prisms", "cylinders", "bullets"):
        return scenes.Scene(kind, [getattr(scenes, kind)(n, seed=seed)])
    if kind == "terrain":
        # Columns and levels whose product is near the size, over a mesh that reaches past them.
        cols = max(4, min(32, int(round(n ** (1.0 / 3.0)))))
        levels = max(1, n // (cols * cols))
        cells = 8 * cols
        return scenes.Scene(kind, [scenes.terrain(cells=cells, cols=cols, levels=levels, top=2.0 + 1.87 * (levels - 1),
                                                  seed=seed)])
    if kind == "planar":
        cols = max(4, int(round(46 * math.sqrt(n / 16384.0))))
        rows = (n + cols - 1) // cols
        return scenes.Scene(kind, [scenes.planar(n=n, cols=cols, spheres=n // 64, seed=seed,
                                                 sphere_height=(10.0, 10.0 + 1.7 * rows))])
    if kind == "uneven":
        # The world sizes are the workload's own; the seed makes what is in the worlds.
        sizes = scenes.config4_bodies(n)
        return scenes.Scene(kind, [scenes.config4(n, seed, int(c), int(c), only=[w]).worlds[0] for w, c in enumerate(sizes)])
    if kind in ("impact", "adjoint"):
        return scenes.config5(n, seed=seed)
    if kind == "jointed":
        return scenes.Scene(kind, [scenes.jointed([seed, w]) for w in range(n)])
    raise ValueError(kind)


class Rollout:
    """A batch, the forces of its frames and the pinned buffers its poses are read into."""

    def __init__(self, case, seed):
        scene = _scene(case, seed)
        self.batch = Batch.from_scene(scene)
        self.frames, self.per_call, self.graph = case["frames"], case["per_call"], case["graph"]
        total = int(self.batch.offsets[-1])
        self.forces = None
        if case["forces"]:
            f = np.random.default_rng([seed, 11]).uniform(-1.0, 1.0, size=(total, 3)).astype(np.float32)
            self.forces = torch.from_numpy(f).pin_memory().numpy()
        self.poses = [(torch.zeros((total, 3)).pin_memory().numpy(), torch.zeros((total, 4)).pin_memory().numpy())
                      for _ in range(2)]
        for _ in range(case["warm"] // self.per_call):
            self.batch.step_checked(DT, self.per_call, graph=self.graph)
        # The state to roll out from. A rollout that outgrows the batch's lists lays the batch out again and so
        # ends its snapshots; the lists have their size after the first one that does not.
        for _ in range(6):
            self.batch.save_state()
            self.roll()
            try:
                self.batch.restore_state()
                return
            except Exception:
                continue
        raise RuntimeError("the batch's lists kept growing")

    def roll(self):
        b = self.batch
        for k in range(self.frames):
            if self.forces is not None:
                b.add_forces(self.forces)
            b.step_checked(DT, self.per_call, graph=self.graph)
            b.read_poses_async(*self.poses[k & 1])
        b.poses_wait()
        return self.poses[(self.frames - 1) & 1]

    def run(self):
        self.batch.restore_state()
        p, q = self.roll()
        return {"positions": p, "rotations": q}


class Adjoint:
    """A recorded run of impact worlds, ready for the model's forward and the adjoint's backward."""

    def __init__(self, case, seed):
        scene = _scene(case, seed)
        self.batch = Batch.from_scene(scene)
        self.precision = case["precision"]
        # Gradients go back to parameters of the model's own precision.
        self.dtype = np.float32 if self.precision == 32 else np.float64
        self.shapes = sum(len(w.shapes) for w in scene.worlds)
        self.batch.tape_record(DT, case["frames"])
        # The loss: the sum of the boxes' squared final x.
        self.boxes = np.zeros(int(self.batch.offsets[-1]), bool)
        for at in self.batch.offsets[:-1]:
            self.boxes[at + 1:at + 65] = True

    def run(self):
        final = self.batch.adjoint_forward(self.precision)
        grad = np.zeros_like(final)
        grad[self.boxes, 0] = 2.0 * final[self.boxes, 0]
        initial, mass, friction = self.batch.adjoint_backward(grad, self.shapes)
        return {"final": final.astype(self.dtype), "initial": initial.astype(self.dtype),
                "mass": mass.astype(self.dtype), "friction": friction.astype(self.dtype)}


class Candidates:
    """Bounds, growths and flags of one world's bodies on the device, at about three pairs a body."""

    def __init__(self, case, seed):
        n = case["size"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        span = 0.9 * max(n, 2) ** (1.0 / 3.0)

        def rand(*shape):
            return torch.rand(shape, generator=g, device="cuda")

        center, half = (rand(n, 3) - 0.5) * span, 0.2 + 0.3 * rand(n, 3)
        self.lo, self.hi = (center - half).contiguous(), (center + half).contiguous()
        self.grow = 0.02 + 0.05 * rand(n)
        moving = abi.TF_PAIR_LIVE | abi.TF_PAIR_DYNAMIC | abi.TF_PAIR_MOVING
        asleep = abi.TF_PAIR_LIVE | abi.TF_PAIR_DYNAMIC
        self.flags = torch.where(rand(n) < 0.9, moving, asleep).to(torch.int32)
        self.capacity = 16 * n
        self.keys = torch.zeros(self.capacity, dtype=torch.int64, device="cuda")
        self.count = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.lib = abi.load()

    def run(self):
        abi.check(self.lib.tf_candidates_noalloc(
            self.lo.data_ptr(), self.hi.data_ptr(), self.grow.data_ptr(), self.flags.data_ptr(), self.flags.numel(),
            self.keys.data_ptr(), self.capacity, self.count.data_ptr(),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)), self.lib)
        return {"keys": self.keys, "count": self.count}


def prepare(case, seed):
    if case["kind"] == "adjoint":
        return Adjoint(case, seed)
    if case["kind"] == "candidates":
        return Candidates(case, seed)
    return Rollout(case, seed)


def run(state):
    return state.run()


# Bodies of a case, and the contacts a body has in it once the scene has come together (about).
CONTACTS = {"boxes": 1.5, "pyramid": 2.8, "hulls": 1.0, "prisms": 1.0, "cylinders": 1.0, "bullets": 0.5, "terrain": 0.7,
            "planar": 0.7, "uneven": 0.4, "impact": 2.7, "adjoint": 2.7, "jointed": 0.3}
UNEVEN_MEAN = 121  # bodies of a world with a log-uniform count from 8 to 512


def _bodies(case):
    kind, n = case["kind"], case["size"]
    if kind == "pyramid":
        return n * (n + 1) // 2 + 1
    return n * {"uneven": UNEVEN_MEAN, "impact": 66, "adjoint": 66, "jointed": 26}.get(kind, 1) + 1


def work(case):
    """Per step, each body read and written once (160 bytes), each shape read once (84), and each candidate (16),
    contact (64) and contact point (84; 2.6 a contact) read and written once; then the poses out. Operations: three
    passes a substep over three rows of a point, about 60 operations each, and about 300 a body."""
    if case["kind"] == "candidates":
        n = case["size"]
        return {"bytes": n * 32 + 3 * n * 8 + 4, "flops": 12 * 3 * n}
    bodies = _bodies(case)
    contacts = CONTACTS[case["kind"]] * bodies
    points = 2.6 * contacts
    steps = case["frames"] * case.get("per_call", 1)
    step_bytes = bodies * (160 + 84) + contacts * (16 + 2 * 64) + points * 2 * 84
    step_flops = 4 * (points * 3 * 3 * 60 + bodies * 300)
    if case["kind"] == "adjoint":
        scale = case["precision"] // 32
        return {"bytes": 3 * steps * step_bytes * scale, "flops": 4 * steps * step_flops}
    return {"bytes": steps * step_bytes + case["frames"] * bodies * (28 + (12 if case["forces"] else 0)),
            "flops": steps * step_flops}


def exact(case, seed):
    """No value in 64 bits: see above."""
    return None
