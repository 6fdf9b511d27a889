"""The workloads this library's speed is measured on.

Every case is one call (or one horizon of calls) that a user's program makes
through the public Python API: a rollout advance of an articulated world or of
a free-body pile, a batch of several worlds, a policy-driven advance through
the task layer, or an advance whose contacts are solved to convergence.

A pass starts from the case's own state (an advance resets every environment
on its first control step), so that repeated passes do the same work: that is
how a sampling controller or a learner with fixed-length episodes calls it.
Start states are made from the seed alone, never by running the library:
trees stand or lie on the ground with their lowest collider touching it, and
piles are columns of bodies resting on each other.
"""

from __future__ import annotations

import ctypes as ct
import math

import numpy as np
import torch

import numi_lab_b200 as nb
from numi_lab_b200 import task as task_layer

MODEL_SEED = 2026          # the benchmark's tree and chain worlds
SUBSTEPS, ITERATIONS, CONTROL_DT = 4, 8, 0.02
CHAIN_DT = 0.005
SCENES = ("pile", "pile_gjk", "cylinder_pile", "hull_pile")
MIX_BODIES = (12, 24, 40, 61)  # body counts of the mix's pile worlds
# Body counts whose worlds have well-conditioned start states: a few others
# hold two boxes, or a cylinder and a sphere, whose contact points rounding
# alone would choose.
BODIES = (8, 9, 11, 12, 14, 17, 20, 23, 25, 28, 35, 36, 41, 44, 47, 49, 53, 56, 61)
CYLINDER_BODIES = (11, 14, 23)
EXACT_TREE_ENV_STEPS = 1000    # about 20 s of the 64-bit restatement below
# Values of include/numi_b200.h.
SPHERE, CAPSULE, BOX, PLANE, CYLINDER, CONVEX = range(6)
FLOATING_ROOT, IMPLICIT_POSITION = 1, 1
ACTUATED, POSITION_LIMIT, VELOCITY_LIMIT, DRIVE = 2, 4, 8, 32


def listed() -> list[dict]:
    return [
        # One robot in a control loop: the latency of one control step.
        {"name": "tree29_one", "kind": "tree", "envs": 1, "steps": 1, "precision": "fp32"},
        # The benchmark's batch of humanoids.
        {"name": "tree29_batch", "kind": "tree", "envs": 4096, "steps": 4, "precision": "fp32"},
        # An odd number of environments in the compensated precision mode.
        {"name": "tree29_compensated", "kind": "tree", "envs": 301, "steps": 3, "precision": "compensated"},
        # The reference-shaped call: host actions in, results in host memory.
        {"name": "tree29_host", "kind": "tree_host", "envs": 1000, "steps": 4, "precision": "fp32"},
        # Contacts solved to convergence: data generation, reference rollouts.
        {"name": "tree29_quality", "kind": "quality", "envs": 256, "steps": 1},
        # Free motion of a fixed-base arm over many short steps.
        {"name": "chain7_free", "kind": "chain", "envs": 1024, "steps": 20},
        # A few small piles: one scene being watched or scripted.
        {"name": "pile9_few", "kind": "scene", "source": "pile", "bodies": 9, "envs": 5, "steps": 1},
        # The pile benchmark's size: 16,384 piles of boxes, spheres, capsules.
        {"name": "pile36_batch", "kind": "scene", "source": "pile", "bodies": 36, "envs": 16384, "steps": 1},
        # Cylinders among the bodies (GJK / EPA pairs).
        {"name": "cylinders23", "kind": "scene", "source": "cylinder_pile", "bodies": 23, "envs": 3000, "steps": 1},
        # Convex hulls among the bodies.
        {"name": "hulls49", "kind": "scene", "source": "hull_pile", "bodies": 49, "envs": 1500, "steps": 1},
        # Chains, trees and piles of several sizes in one launch.
        {"name": "mix", "kind": "mix", "envs": 4000, "steps": 3},
        # A learner's collection step: policy, task layer, transitions.
        {"name": "policy_task", "kind": "policy", "envs": 2048, "steps": 8},
    ]


def draw(rng) -> dict:
    """One more case: the kinds in proportion to their use, sizes spread over
    the logarithm of their range, the cost of a case bounded by the largest
    listed one of its kind."""

    def log(lo: float, hi: float) -> int:
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tree", "tree", "tree", "scene", "scene", "scene", "tree_host", "quality", "chain", "mix", "policy"])
    if kind in ("tree", "tree_host"):
        steps = log(1, 4)
        envs = log(1, 16384 // steps)
        return {"kind": kind, "envs": envs, "steps": steps, "precision": rng.choice(["fp32", "fp32", "fp64-inertia", "compensated"])}
    if kind == "quality":
        return {"kind": kind, "envs": log(1, 256), "steps": 1}
    if kind == "chain":
        return {"kind": kind, "envs": log(1, 16384), "steps": log(1, 20)}
    if kind == "mix":
        return {"kind": kind, "envs": log(10, 4000), "steps": log(1, 3)}
    if kind == "policy":
        return {"kind": kind, "envs": log(1, 2048), "steps": log(1, 8)}
    source = rng.choice(SCENES)
    bodies = rng.choice(CYLINDER_BODIES if source == "cylinder_pile" else BODIES)
    most = 500000 if source == "pile" else 36000
    return {"kind": kind, "source": source, "bodies": bodies, "envs": log(1, most // bodies), "steps": 1}


def scene_substeps(source: str) -> int:
    """Cylinder and hull piles take one 5 ms step per control step: every
    substep's support-mapped pairs amplify the rounding of the one before."""

    return 1 if source in ("cylinder_pile", "hull_pile") else SUBSTEPS


def work(case: dict) -> dict:
    """Bytes: resident state read and written once a pass, each control step's
    actions read and observations and status written once.  Flops: the
    articulated-body sweeps, contact rows and solver sweeps of every substep."""

    envs, steps = case["envs"], case["steps"]

    def articulated(n, nq, nv, na, bodies, manifolds, contacts, substeps):
        state = 8 * (nq + nv) + 2 * 224 * manifolds
        flops = 1400 * bodies + contacts * (3 * 12 * 12 + (ITERATIONS + 1) * 3 * 12 * 4 + 400 + 24 * contacts)
        return np.array([n * (state + steps * 4 * (na + nq + nv + 1)), n * steps * substeps * flops], np.float64)

    def scene(n, bodies, substeps=SUBSTEPS):
        flops = 200 * bodies + 8 * bodies * bodies + 2.5 * bodies * (900 + (ITERATIONS + 1) * 120)
        return np.array([n * bodies * (8 * 13 + 2 * 228 + steps * 4 * 13), n * steps * substeps * flops], np.float64)

    def tree(n):
        return articulated(n, 36, 35, 29, 30, 14, 16, SUBSTEPS)

    def chain(n):
        return articulated(n, 7, 7, 7, 7, 0, 0, 1)

    if case["kind"] == "scene":
        total = scene(envs, case["bodies"], scene_substeps(case["source"]))
    elif case["kind"] == "chain":
        total = chain(envs)
    elif case["kind"] == "mix":
        n_chain, n_tree, n_pile = mix_counts(envs)
        total = chain(n_chain) + tree(n_tree) + sum(scene(n, b) for n, b in zip(n_pile, MIX_BODIES))
    else:
        total = tree(envs)
        if case["kind"] == "quality":  # about ten Newton steps, each a 35 x 35 factorisation
            total[1] += envs * steps * SUBSTEPS * 10 * (35 ** 3 / 3 + 16 * 9 * 12 * 12 * 2)
        if case["kind"] == "policy":  # actor 99-256-128-29, critic 99-64-1; latents, values, transitions
            weights = 99 * 256 + 256 * 128 + 128 * 29 + 99 * 64 + 64
            total += np.array([4 * weights + envs * steps * 4 * (29 + 2 + 32 + 28), envs * steps * 2 * weights])
    return {"bytes": float(total[0]), "flops": float(total[1])}


# Measured as the library's three precision modes (other orders and widths of
# the same sums) and inputs moved by half an ulp differ: 4e-6 for chains, 1e-6
# to 2e-5 for contact worlds in bulk, times about four.  A contact world may
# also see one environment among thousands take another contact decision (a
# point kept or dropped), which alone reaches 1e-3 of the whole.
def tolerance(case: dict) -> dict:
    if case["kind"] == "chain":
        return {"rel": 3e-5, "max": 5e-3}
    return {"rel": 4e-3, "max": 0.9, "differ": 0.01}


# -- inputs --------------------------------------------------------------


def mix_counts(envs: int) -> tuple[int, int, list[int]]:
    """40 % chains, 30 % trees, the rest piles over MIX_BODIES."""

    n_chain, n_tree = max(1, int(0.4 * envs)), max(1, int(0.3 * envs))
    rest = max(len(MIX_BODIES), envs - n_chain - n_tree)
    return n_chain, n_tree, [rest * (i + 1) // len(MIX_BODIES) - rest * i // len(MIX_BODIES) for i in range(len(MIX_BODIES))]


_SEEDS: dict[int, int] = {}


def scene_seed(bodies: int) -> int:
    """A model seed whose pile has this many bodies."""

    if bodies not in _SEEDS:
        _SEEDS.update(nb.world.pile_seeds_by_body_count([bodies]))
    return _SEEDS[bodies]


def quat_mul(a: np.ndarray, b: np.ndarray) -> np.ndarray:
    ax, ay, az, aw = np.moveaxis(a, -1, 0)
    bx, by, bz, bw = np.moveaxis(b, -1, 0)
    return np.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                     aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], -1)


def rotation(q: np.ndarray) -> np.ndarray:
    """Rotation matrices [..., 3, 3] of unit quaternions xyzw."""

    x, y, z, w = np.moveaxis(q, -1, 0)
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).reshape(*q.shape[:-1], 3, 3)


def tilts(rng, shape, sigma: float) -> np.ndarray:
    """Small random rotations: no box face, cylinder cap or foot lies exactly flat."""

    half = 0.5 * rng.normal(0.0, sigma, (*shape, 3))
    q = np.concatenate([half, np.ones((*shape, 1))], -1)
    return q / np.linalg.norm(q, axis=-1, keepdims=True)


def tree_inputs(envs: int, steps: int, seed: int):
    """Start state (half standing, half lying on the back or the front, the
    lowest collider within half a millimetre of the ground) and drive targets
    N(0, 0.3)."""

    rng = np.random.default_rng(seed)
    tree = Tree(nb.world.compile_model("tree29", MODEL_SEED))
    q = np.zeros((envs, tree.nq))
    q[:, 7:] = rng.normal(0.0, 0.15, (envs, tree.nq - 7))
    pitch = np.where(rng.random(envs) < 0.5, rng.normal(0.0, 0.05, envs), rng.choice([-0.5, 0.5], envs) * math.pi)
    yaw = rng.uniform(-math.pi, math.pi, envs)
    zero = np.zeros(envs)
    q[:, 3:7] = quat_mul(quat_mul(np.stack([zero, zero, np.sin(yaw / 2), np.cos(yaw / 2)], -1),
                                  np.stack([zero, np.sin(pitch / 2), zero, np.cos(pitch / 2)], -1)), tilts(rng, (envs,), 0.05))
    q[:, 2] = -tree.lowest(q) + rng.uniform(-5e-4, 5e-4, envs)
    v = rng.normal(0.0, 0.1, (envs, tree.nv))
    actions = rng.normal(0.0, 0.3, (steps, envs, tree.nv - 6))
    return q.astype(np.float32), v.astype(np.float32), actions.astype(np.float32)


def chain_inputs(envs: int, steps: int, seed: int):
    """Joint angles U(-pi/2, pi/2), rates N(0, 1), torques N(0, 5)."""

    rng = np.random.default_rng(seed + 1)
    return (rng.uniform(-math.pi / 2, math.pi / 2, (envs, 7)).astype(np.float32), rng.normal(0.0, 1.0, (envs, 7)).astype(np.float32),
            rng.normal(0.0, 5.0, (steps, envs, 7)).astype(np.float32))


def scene_inputs(source: str, bodies: int, envs: int, seed: int):
    """Columns of one or two bodies in rows whose neighbours almost touch;
    every body rests within half a millimetre on the ground or on the body
    below."""

    rng = np.random.default_rng(seed + 2)
    rec = nb.world.compile_model(source, scene_seed(bodies))
    q = np.zeros((envs, bodies, 7))
    v = rng.normal(0.0, 0.02, (envs, bodies, 6))
    wide = np.zeros((envs, bodies))                          # horizontal reach
    low, high = np.zeros((envs, bodies)), np.zeros((envs, bodies))  # extent below and above the centre
    yaw = rng.uniform(-math.pi, math.pi, (envs, bodies))
    turn = np.stack([0 * yaw, 0 * yaw, np.sin(yaw / 2), np.cos(yaw / 2)], -1)
    upright = np.array([math.sqrt(0.5), 0.0, 0.0, math.sqrt(0.5)])
    for b in range(bodies):
        if rec.shapes[b].shape_type == CYLINDER:  # standing in about half of the environments, else lying
            up = rng.random(envs) < 0.5
            turn[up, b] = quat_mul(turn[up, b], np.broadcast_to(upright, (int(up.sum()), 4)))
    q[..., 3:] = quat_mul(turn, tilts(rng, (envs, bodies), 0.01))
    R = rotation(q[..., 3:])
    for b in range(bodies):
        s, up = rec.shapes[b], R[:, b, 2, :]  # world z in the body's frame
        d = vec(s.dimensions)
        if s.shape_type == BOX:
            low[:, b] = high[:, b] = np.abs(up) @ d
            wide[:, b] = math.hypot(d[0], d[1])
        elif s.shape_type == CONVEX:
            points = rec.hull_vertices[s.hull_first:s.hull_first + s.hull_count, :3].astype(np.float64) * d
            height = up @ points.T
            low[:, b], high[:, b], wide[:, b] = -height.min(1), height.max(1), np.linalg.norm(points, axis=1).max()
        elif s.shape_type == CYLINDER:
            axial, across = np.abs(up[:, 1]), np.sqrt(1.0 - up[:, 1] ** 2)
            low[:, b] = high[:, b] = axial * d[1] + across * d[0]
            wide[:, b] = across * d[1] + d[0]
        else:  # spheres (no length) and capsules
            length = d[1] if s.shape_type == CAPSULE else 0.0
            low[:, b] = high[:, b] = np.abs(up[:, 1]) * length + d[0]
            wide[:, b] = length + d[0]
    # A lighter box stands on a heavier one, a sphere on any other body: a
    # capsule, cylinder or hull lying flat on a box would leave the choice of
    # its contact points to rounding.
    def heaviest(*types):
        return sorted((b for b in range(bodies) if rec.shapes[b].shape_type in types), key=lambda b: -rec.bodies[b].mass_inverse_mass[0])

    boxes, spheres = heaviest(BOX), heaviest(SPHERE)
    stacks = [[b] for b in boxes[:-(-len(boxes) // 2)]]
    for under, b in zip(stacks, boxes[len(stacks):]):
        under.append(b)
    others = [[b] for b in heaviest(CAPSULE, CYLINDER, CONVEX)]
    for k, b in enumerate(spheres):
        others[k].append(b) if k < len(others) else others.append([b])
    stacks += others
    columns = len(stacks)
    side = max(1, int(round(math.sqrt(columns))))
    top = np.zeros((envs, columns))
    reach = np.stack([wide[:, stack].max(1) for stack in stacks], 1) + 0.003
    x, y = np.zeros((envs, columns)), np.zeros((envs, columns))
    depth = np.zeros(envs)
    for first in range(0, columns, side):
        tall = reach[:, first:first + side].max(1)
        at = np.zeros(envs)
        for c in range(first, min(first + side, columns)):
            x[:, c], y[:, c] = at + reach[:, c], depth + tall
            at = at + 2 * reach[:, c]
        depth = depth + 2 * tall
    for c, stack in enumerate(stacks):
        for b in stack:
            q[:, b, 0] = x[:, c] + rng.normal(0.0, 0.001, envs)
            q[:, b, 1] = y[:, c] + rng.normal(0.0, 0.001, envs)
            q[:, b, 2] = top[:, c] + low[:, b] + rng.uniform(-5e-4, 5e-4, envs)
            top[:, c] += low[:, b] + high[:, b]
    return q.reshape(envs, -1).astype(np.float32), v.reshape(envs, -1).astype(np.float32)


# -- prepare and run -----------------------------------------------------


def first_step_resets(steps: int, envs: int) -> torch.Tensor:
    mask = torch.zeros((steps, envs), dtype=torch.int32, device="cuda")
    mask[0] = 1
    return mask


def world_of(source: str, envs: int, model_seed: int, seed: int, **options):
    """A world whose friction scales and reset draws come from `seed`."""

    world = nb.World(source, envs, seed=model_seed, **options)
    world.reset(seed)
    return world


def contact_options(substeps: int = SUBSTEPS) -> dict:
    return {"substeps": substeps, "velocity_iterations": ITERATIONS, "control_dt": CONTROL_DT / SUBSTEPS * substeps}


def articulated_part(source: str, envs: int, steps: int, seed: int, **options) -> dict:
    if source == "chain7":
        q, v, actions = chain_inputs(envs, steps, seed)
        world = world_of(source, envs, MODEL_SEED, seed, substeps=1, control_dt=CHAIN_DT, **options)
    else:
        q, v, actions = tree_inputs(envs, steps, seed)
        world = world_of(source, envs, MODEL_SEED, seed, **contact_options(), **options)
    world.set_state(q, v, as_reset_state=True)
    return {"world": world, "host_actions": actions, "actions": torch.from_numpy(actions).cuda()}


def scene_part(source: str, bodies: int, envs: int, steps: int, seed: int) -> dict:
    world = world_of(source, envs, scene_seed(bodies), seed, **contact_options(scene_substeps(source)))
    q, v = scene_inputs(source, bodies, envs, seed)
    world.set_state(q, v, as_reset_state=True)
    return {"world": world, "actions": torch.zeros((steps, envs, 0), device="cuda")}


def dense_layers(rng, sizes, activations):
    return [(rng.normal(0.0, 1.0 / math.sqrt(a), (b, a)).astype(np.float32), rng.normal(0.0, 0.1, b).astype(np.float32), f)
            for (a, b), f in zip(zip(sizes[:-1], sizes[1:]), activations)]


def prepare(case: dict, seed: int) -> dict:
    envs, steps, kind = case["envs"], case["steps"], case["kind"]
    state = {"kind": kind, "steps": steps}
    if kind == "mix":
        n_chain, n_tree, n_pile = mix_counts(envs)
        parts = [articulated_part("chain7", n_chain, steps, seed), articulated_part("tree29", n_tree, steps, seed)]
        parts += [scene_part("pile_gjk", b, n, steps, seed) for n, b in zip(n_pile, MIX_BODIES)]
        state["worlds"] = [p["world"] for p in parts]
        state["actions"] = [p["actions"] for p in parts]
        state["masks"] = [first_step_resets(steps, w.envs) for w in state["worlds"]]
        state["status"] = [torch.zeros((steps, w.envs), dtype=torch.int32, device="cuda") for w in state["worlds"]]
        state["batch"] = nb.Batch(state["worlds"])
        return state
    if kind == "scene":
        state.update(scene_part(case["source"], case["bodies"], envs, steps, seed))
    elif kind == "policy":
        state.update(articulated_part("tree29", envs, steps, seed))
        world, rng = state["world"], np.random.default_rng(seed + 3)
        default_q = np.zeros(world.nq, np.float32)
        default_q[2] = nb.sample_reset("tree29", MODEL_SEED, MODEL_SEED, 0, 1)[0][0, 2]
        default_q[6] = 1.0
        world.set_task(task_layer.locomotion_task(world.model(), default_q, maximum_episode_steps=500, noise=0.01))
        frame, na = world.observation_count, world.action_count
        world.set_policy(layers=dense_layers(rng, [frame, 256, 128, na], ["elu", "silu", "tanh"]),
                         critic_layers=dense_layers(rng, [frame, 64, 1], ["relu", "identity"]), revision=1, action_clip=2.5,
                         observation_mean=np.zeros(frame, np.float32), observation_inverse_std=np.ones(frame, np.float32),
                         observation_clip=10.0, action_scale=np.full(na, 0.5, np.float32), action_log_std=np.full(na, -1.5, np.float32))
    else:
        source = "chain7" if kind == "chain" else "tree29"
        state.update(articulated_part(source, envs, steps, seed, precision=case.get("precision", "fp32")))
        if kind == "quality":
            state["world"].set_solver("quality_newton")
    world = state["world"]
    state["mask"] = first_step_resets(steps, envs)
    state["host_mask"] = state["mask"].cpu().numpy().astype(np.uint32)
    if kind == "tree_host":
        world.set_state_readback(True)
    if kind not in ("policy", "tree_host"):
        state["observations"] = torch.zeros((steps, envs, world.observation_count), device="cuda")
        state["status"] = torch.zeros((steps, envs), dtype=torch.int32, device="cuda")
    return state


def final_state(world) -> tuple[np.ndarray, np.ndarray]:
    """q and v of a batched world, as its owner reads them after a horizon."""

    q, v = np.empty((world.envs, world.nq), np.float32), np.empty((world.envs, world.nv), np.float32)
    pointer = ct.POINTER(ct.c_float)
    world._lib.check(world._lib.lib.mr_task_rollout_copy_state(world._handle, q.ctypes.data_as(pointer), v.ctypes.data_as(pointer), None),
                     "copy_state")
    return q, v


def run(state: dict):
    kind = state["kind"]
    if kind == "mix":
        state["batch"].step(state["actions"], state["masks"], state["status"])
        return {"status": state["status"], "state": [list(final_state(w)) for w in state["worlds"]]}
    world = state["world"]
    if kind == "tree_host":
        out = world.advance_host(state["host_actions"], state["host_mask"], raise_on_failure=False)
        return {"observations": out["observations"], "status": out["status"], "contacts": out["contacts"], "final_q": out["final_q"]}
    if kind == "policy":
        observations, status = world.step_policy(state["steps"], reset_mask=state["mask"], wait=False)
        outputs, transitions = world.policy_outputs(), world.transitions(state["steps"])
        return {"observations": observations, "status": status, "policy": outputs,
                "reward": transitions["reward"], "done": transitions["done"].astype(np.int64)}
    world.step(state["actions"], state["mask"], state["observations"], state["status"])
    return {"observations": state["observations"], "status": state["status"]}


# -- 64-bit restatement --------------------------------------------------
# The articulated control step in plain numpy: dense joint-space inertia
# instead of articulated-body sweeps, plane contacts with persistent
# manifolds, the fixed-budget cone iteration or the converged solve.


def cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def vec(c_array, n=3):
    return np.array([float(x) for x in c_array[:n]])


class Tree:
    """One world's bodies, revolute joints, drives and colliders."""

    def __init__(self, rec) -> None:
        w = rec.world
        self.nq, self.nv, self.floating = int(w.nq), int(w.nv), int(w.root_type) == FLOATING_ROOT
        self.implicit = int(w.actuation_mode) == IMPLICIT_POSITION
        self.gravity = vec(w.gravity)
        _, _, self.max_depenetration, self.slop = (float(x) for x in w.solver_scales)
        self.thresholds = [float(x) for x in w.manifold_thresholds]
        self.speculative, self.speed_envelope = float(w.speculative[0]), float(w.speculative[1])
        self.bodies = [rec.bodies[i] for i in range(w.body_count) if rec.bodies[i].articulated]
        self.parent = [-1] + [int(b.parent_body) for b in self.bodies[1:]]
        self.mass = np.array([float(b.mass_inverse_mass[0]) for b in self.bodies])
        self.inertia = np.array([[vec(b.inertia[r]) for r in range(3)] for b in self.bodies])
        self.damping = np.array([[float(b.damping_speed[0]), float(b.damping_speed[1])] for b in self.bodies])
        self.joints = [None] + [rec.joints[b.inbound_joint] for b in self.bodies[1:]]
        self.dofs = [rec.dofs[d] for d in range(self.nv)]
        self.ancestors = [list(range(6)) if self.floating else []]
        for b in range(1, len(self.bodies)):
            self.ancestors.append(self.ancestors[self.parent[b]] + [int(self.joints[b].v_index)])
        self.limits = np.array([[float(x) for x in d.limits] for d in self.dofs])
        self.drive = np.array([[float(x) for x in d.drive] for d in self.dofs])
        self.driven = np.array([bool(d.flags & DRIVE) for d in self.dofs])
        self.velocity_limited = np.array([bool(d.flags & VELOCITY_LIMIT) for d in self.dofs])
        self.position_limited = np.array([bool(d.flags & POSITION_LIMIT) for d in self.dofs])
        self.actuated = np.array([bool(d.flags & ACTUATED) for d in self.dofs])
        self.joint_dofs = slice(6, self.nv) if self.floating else slice(0, self.nv)
        self.joint_q = slice(7, self.nq) if self.floating else slice(0, self.nq)
        self.shapes = [rec.shapes[i] for i in range(w.shape_count) if rec.shapes[i].shape_type != PLANE]
        friction = [rec.materials[i].friction for i in range(w.material_count)]
        self.friction = [math.sqrt(friction[s.material][0] * friction[rec.shapes[w.shape_count - 1].material][0]) for s in self.shapes]
        response = [rec.materials[i].response for i in range(w.material_count)]
        self.restitution = max([float(r[0]) for r in response], default=0.0)
        self.restitution_speed = max([float(r[1]) for r in response], default=0.0)

    def kinematics(self, q, v):
        """Per body: position, orientation, angular and linear velocity, and
        the velocity-product accelerations; per DoF its axis and origin."""

        n, nbodies = q.shape[0], len(self.bodies)
        c, rot = np.zeros((n, nbodies, 3)), np.zeros((n, nbodies, 4))
        w, lin, alpha, acc = (np.zeros((n, nbodies, 3)) for _ in range(4))
        axis, origin = np.zeros((n, self.nv, 3)), np.zeros((n, self.nv, 3))
        rot[:, 0, 3] = 1.0
        if self.floating:
            c[:, 0], rot[:, 0] = q[:, :3], q[:, 3:7] / np.linalg.norm(q[:, 3:7], axis=1, keepdims=True)
            w[:, 0], lin[:, 0] = v[:, 3:6], v[:, :3]
            axis[:, 0:3] = axis[:, 3:6] = np.eye(3)
            origin[:, 3:6] = c[:, None, 0]
        for b in range(1, nbodies):
            p, j = self.parent[b], self.joints[b]
            d, qi = int(j.v_index), int(j.q_index)
            at = quat_mul(rot[:, p], vec(j.parent_rotation, 4))
            unit = vec(j.axis) / np.linalg.norm(vec(j.axis))
            half = 0.5 * q[:, qi]
            turn = np.concatenate([np.sin(half)[:, None] * unit, np.cos(half)[:, None]], 1)
            rb = quat_mul(quat_mul(at, turn), vec(j.child_rotation, 4) * np.array([-1.0, -1.0, -1.0, 1.0]))
            rb /= np.linalg.norm(rb, axis=1, keepdims=True)
            ja = rotation(at) @ unit
            jp = c[:, p] + rotation(rot[:, p]) @ vec(j.parent_anchor)
            ca = rotation(rb) @ vec(j.child_anchor)
            rate, arm = v[:, d, None], jp - c[:, p]
            axis[:, d], origin[:, d] = ja, jp
            c[:, b], rot[:, b] = jp - ca, rb
            w[:, b] = w[:, p] + ja * rate
            lin[:, b] = lin[:, p] + cross(w[:, p], arm) - cross(w[:, b], ca)
            alpha[:, b] = alpha[:, p] + cross(w[:, p], ja) * rate
            acc[:, b] = (acc[:, p] + cross(alpha[:, p], arm) + cross(w[:, p], cross(w[:, p], arm)) - cross(alpha[:, b], ca)
                         - cross(w[:, b], cross(w[:, b], ca)))
        return c, rot, w, lin, alpha, acc, axis, origin

    def columns(self, b, x, axis, origin):
        """Point Jacobian [n, 3, nv] of world point x on body b, and its angular part."""

        jv, jw = np.zeros((x.shape[0], 3, self.nv)), np.zeros((x.shape[0], 3, self.nv))
        for d in self.ancestors[b]:
            if self.floating and d < 3:
                jv[:, :, d] = axis[:, d]
            else:
                jv[:, :, d] = cross(axis[:, d], x - origin[:, d])
                jw[:, :, d] = axis[:, d]
        return jv, jw

    def lowest(self, q):
        """Height of the lowest collider point above the root's origin height."""

        c, rot = self.kinematics(np.asarray(q, np.float64), np.zeros((q.shape[0], self.nv)))[:2]
        low = np.full(q.shape[0], np.inf)
        for s in self.shapes:
            rotm = rotation(rot[:, s.body])
            z = c[:, s.body, 2] + (rotm @ vec(s.local_position))[:, 2]
            d = vec(s.dimensions)
            reach = d[0] if s.shape_type == SPHERE else np.abs(rotm[:, 2, :]) @ d
            low = np.minimum(low, z - reach)
        return low

    def drives(self, q, v, target, h):
        if not self.implicit:
            return np.clip(target, -self.limits[:, 3], self.limits[:, 3])
        position = np.zeros_like(v)
        position[:, self.joint_dofs] = q[:, self.joint_q]
        goal = np.where(self.position_limited, np.clip(target, self.limits[:, 0], self.limits[:, 1]), target)
        tau = self.drive[:, 0] * (goal - position - h * v) - self.drive[:, 1] * v
        return np.where(self.driven, np.clip(tau, -self.limits[:, 3], self.limits[:, 3]), 0.0)

    def dynamics(self, q, v, tau, h):
        """Free velocity after h, the joint-space inertia and the kinematics."""

        kin = self.kinematics(q, v)
        c, rot, w, lin, alpha, acc, axis, origin = kin
        n = q.shape[0]
        H, force = np.zeros((n, self.nv, self.nv)), np.array(tau)
        for b in range(1 if not self.floating else 0, len(self.bodies)):
            jv, jw = self.columns(b, c[:, b], axis, origin)
            R = rotation(rot[:, b])
            I = R @ self.inertia[b] @ np.swapaxes(R, 1, 2)
            H += self.mass[b] * np.swapaxes(jv, 1, 2) @ jv + np.swapaxes(jw, 1, 2) @ I @ jw
            momentum = (I @ w[:, b, :, None])[..., 0]
            f = self.mass[b] * (acc[:, b] - self.gravity) + self.damping[b, 0] * lin[:, b]
            t = (I @ alpha[:, b, :, None])[..., 0] + cross(w[:, b], momentum) + self.damping[b, 1] * w[:, b]
            force -= (np.swapaxes(jv, 1, 2) @ f[..., None] + np.swapaxes(jw, 1, 2) @ t[..., None])[..., 0]
        armature = self.drive[:, 2] + (np.where(self.driven, h * self.drive[:, 1] + h * h * self.drive[:, 0], 0.0) if self.implicit else 0.0)
        H += np.diag(armature)
        return v + h * np.linalg.solve(H, force[..., None])[..., 0], H, kin

    def integrate(self, q, v, h):
        q = q.copy()
        q[:, self.joint_q] += h * v[:, self.joint_dofs]
        if self.floating:
            q[:, :3] += h * v[:, :3]
            turn = h * v[:, 3:6]
            angle = np.linalg.norm(turn, axis=1, keepdims=True)
            s = np.where(angle > 1e-6, np.sin(0.5 * angle) / np.maximum(angle, 1e-300), 0.5 - angle * angle / 48)
            r = quat_mul(np.concatenate([turn * s, np.cos(0.5 * angle)], 1), q[:, 3:7])
            q[:, 3:7] = r / np.linalg.norm(r, axis=1, keepdims=True)
        return q


PAD = 0.00000762939453125  # of the collision queries and bounds, relative to the scale
DOWN = np.array([0.0, 0.0, -1.0])  # contact normal, from the tree's collider to the ground


def plane_manifold(tree, s, old, body, R, margin):
    """The persistent manifold of one collider on the ground: points (local
    anchor, ground anchor, feature, impulse), at most four, and its tangent
    in the body's frame.  `old` is the last substep's, or None."""

    shape = tree.shapes[s]
    d, local = vec(shape.dimensions), vec(shape.local_position)
    center = body + R @ local
    offset = float(shape.contact_rest_bound[0])
    if shape.shape_type == SPHERE:
        surfaces, extent, size = [center + d[0] * DOWN], np.full(3, d[0]), d[0]
    else:
        surfaces = [center + R @ (d * [1 if i & 1 else -1, 1 if i & 2 else -1, 1 if i & 4 else -1]) for i in range(8)]
        extent, size = np.abs(R) @ d, d.max()
    lower, upper = center - extent - offset, center + extent + offset
    inflate = (np.maximum(np.abs(lower), np.abs(upper)) + 1.0) * PAD + margin
    scale = max(np.abs(center).max(), size, offset + margin, np.abs(lower - inflate).max(), np.abs(upper + inflate).max())
    accepted = offset + margin + (scale + 1.0) * PAD
    raw = [(i, x) for i, x in enumerate(surfaces) if x[2] <= accepted]
    if not raw:
        return None
    brk, drift, merge, cosine = tree.thresholds
    found, tangent = [], None
    if old is not None and (R @ old["normal"]) @ DOWN >= cosine:
        moved = R @ old["tangent"]
        tangent = moved - DOWN * (moved @ DOWN)
        for p in old["points"]:
            delta = p["ground"] - (body + R @ p["anchor"])
            sep = delta @ DOWN
            if sep <= brk and np.linalg.norm(delta - DOWN * sep) <= drift:
                found.append(dict(p, sep=sep, world=0.5 * (body + R @ p["anchor"] + p["ground"]), fresh=False))
    for i, x in raw:
        ground = x * [1.0, 1.0, 0.0]
        new = {"anchor": R.T @ (x - body), "ground": ground, "feature": i, "sep": x[2], "world": 0.5 * (x + ground)}
        match = next((k for k, p in enumerate(found) if p["feature"] == i), None)
        if match is None:
            match = next((k for k, p in enumerate(found) if ((p["anchor"] - new["anchor"]) ** 2).sum() +
                          ((p["ground"] - ground) ** 2).sum() <= 2 * merge * merge), None)
        if match is None:
            found.append(dict(new, impulse=np.zeros(3), fresh=True))
        else:
            found[match] = dict(new, impulse=found[match]["impulse"], fresh=found[match]["fresh"])
    if len(found) > 4:
        found.sort(key=lambda p: (p["sep"], p["feature"]))
        chosen, rest = found[:1], found[1:]
        for stage in (1, 2, 3):
            best, best_score = None, -1.0
            for p in rest:
                flat = [(p["world"] - k["world"]) * [1, 1, 0] for k in chosen]
                if stage == 2:
                    score = abs(cross(chosen[1]["world"] - chosen[0]["world"], p["world"] - chosen[0]["world"])[2])
                else:
                    score = min(f @ f for f in flat)
                tie = max(1e-12, 1e-5 * max(abs(score), abs(best_score)))
                if score > best_score + tie or (abs(score - best_score) <= tie and (best is None or p["feature"] < best["feature"])):
                    best, best_score = p, score
            chosen.append(best)
            rest = [p for p in rest if p is not best]
        found = chosen
    found.sort(key=lambda p: p["feature"])
    if tangent is None or tangent @ tangent <= 1e-12:
        tangent = np.array([0.0, 1.0, 0.0])
    return {"points": found, "normal": R.T @ DOWN, "tangent": R.T @ (tangent / np.linalg.norm(tangent))}


def cone(p, mu):
    """The impulse's projection as the fixed-budget iteration makes it."""

    p = np.array(p)
    p[:, 0] = np.maximum(p[:, 0], 0.0)
    limit, slip = mu * p[:, 0], np.hypot(p[:, 1], p[:, 2])
    p[:, 1:] *= np.where(slip > limit, np.where(limit > 0, limit / np.maximum(slip, 1e-300), 0.0), 1.0)[:, None]
    return p


def cone_sweeps(W, u_free, target, mu, warm, iterations):
    """Block-Jacobi sweeps with the relaxed, regularised block inverses."""

    n = len(mu)
    blocks = W.reshape(n, 3, n, 3)
    diag = np.abs(blocks[np.arange(n), 0, np.arange(n), 0])
    rows = np.abs(blocks[:, 0, :, 0]).sum(1)
    relax = np.where(rows > np.maximum(diag, 1e-10), np.clip(diag / rows, 1 / 32, 1.0), 1.0)
    inverse = []
    for c in range(n):
        m = blocks[c, :, c, :]
        scale = np.abs(m).max()
        inverse.append(np.linalg.inv(0.5 * (m + m.T) / scale + 0.01 * np.eye(3)) / scale)
    inverse, lam = np.array(inverse), cone(warm, mu)
    for _ in range(iterations):
        u = u_free + (W @ lam.reshape(-1)).reshape(n, 3)
        step = cone(lam + (inverse @ (target - u)[..., None])[..., 0], mu) - lam
        lam = lam + relax[:, None] * step
    return lam


def converged_impulses(H, G, u_free, target, mu, regularization=1e-6):
    """argmin 0.5 l'(G H^-1 G' + r I)l + (u_free - target)'l over the friction
    cones: Newton on the factor-space primal, with a continuation on r."""

    n, nv = len(mu), H.shape[0]
    Y = np.linalg.solve(np.linalg.cholesky(H), G.T)
    b = (u_free - target).reshape(-1)
    z = np.zeros(nv)

    def project(a):
        """Euclidean projection on the cones, and its derivative."""
        out, jac = np.zeros((n, 3)), np.zeros((n, 3, 3))
        for c in range(n):
            x, t, m = a[c, 0], a[c, 1:], mu[c]
            s = np.linalg.norm(t)
            if s <= m * x:
                out[c], jac[c] = a[c], np.eye(3)
            elif x + m * s > 0:
                g = np.concatenate([[1.0], m * t / s])
                k = (x + m * s) / (1 + m * m)
                out[c], jac[c] = k * g, np.outer(g, g) / (1 + m * m)
                e = np.array([0.0, -t[1] / s, t[0] / s])
                jac[c] += k * m / s * np.outer(e, e)
        return out, jac

    for r in (3000 * regularization, 30 * regularization, regularization):
        def gradient(z):
            lam, jac = project(-(b + Y.T @ z).reshape(n, 3) / r)
            return z - Y @ lam.reshape(-1), lam, jac

        def value(z):
            lam, _ = project(-(b + Y.T @ z).reshape(n, 3) / r)
            return 0.5 * z @ z + 0.5 * r * (lam * lam).sum()

        g, lam, jac = gradient(z)
        for _ in range(200):
            if np.abs(g).max() <= 1e-13 * (1 + np.abs(z).max()):
                break
            K = np.eye(nv)
            for c in range(n):
                Yc = Y[:, 3 * c:3 * c + 3]
                K += Yc @ jac[c] @ Yc.T / r
            step, t, f0 = -np.linalg.solve(K, g), 1.0, value(z)
            while t > 1e-10 and value(z + t * step) > f0 + 1e-4 * t * (g @ step) + 1e-15 * abs(f0):
                t *= 0.5
            if t <= 1e-10:
                break
            z = z + t * step
            g, lam, jac = gradient(z)
    return lam


def contact_substep(tree, q, v, vf, H, kin, manifolds, friction, h, quality):
    """One environment's contact solve: the velocity after it, and the new manifolds."""

    c, rot, _, _, _, _, axis, origin = kin
    speed = np.abs(vf).sum()
    rows, u_free, target, mu, where = [], [], [], [], []
    new = {}
    for s, shape in enumerate(tree.shapes):
        bodyid = int(shape.body)
        margin = tree.speculative * min(h * speed * max(float(shape.contact_rest_bound[2]), 0.25), h * tree.speed_envelope)
        R, body = rotation(rot[bodyid]), c[bodyid]
        m = plane_manifold(tree, s, manifolds.get(s), body, R, margin)
        if m is None:
            continue
        new[s] = m
        tangent = R @ m["tangent"]
        tangent -= DOWN * (tangent @ DOWN)
        tangent /= np.linalg.norm(tangent)
        frame = np.stack([DOWN, tangent, cross(DOWN, tangent)])
        for p in m["points"]:
            x = body + R @ p["anchor"]
            point, sep = 0.5 * (x + p["ground"]), (p["ground"] - x) @ DOWN
            jac = -frame @ tree.columns(bodyid, point[None], axis[None], origin[None])[0][0]
            u = jac @ vf
            goal = -sep / h if sep > 0 else 0.0
            stab = min(max(-h * min(sep + tree.slop, 0.0) / (4 * h * h * 2.25), 0.0), tree.max_depenetration)
            if p["fresh"] and u[0] - goal < -tree.restitution_speed:
                stab = max(stab, -tree.restitution * (u[0] - goal))
            rows.append(jac)
            u_free.append(u)
            target.append([goal + stab, 0.0, 0.0])
            mu.append(tree.friction[s] * friction)
            where.append(p)
    v = vf.copy()
    if rows:
        G, u_free, target, mu = np.concatenate(rows), np.array(u_free), np.array(target), np.array(mu)
        Hinv_G = np.linalg.solve(H, G.T)
        if quality:
            lam = converged_impulses(H, G, u_free, target, mu)
        else:
            lam = cone_sweeps(G @ Hinv_G, u_free, target, mu, np.array([p["impulse"] for p in where]), ITERATIONS)
        v = v + Hinv_G @ lam.reshape(-1)
        for p, impulse in zip(where, lam):
            p["impulse"] = impulse
    v = np.where(tree.velocity_limited, np.clip(v, -tree.limits[:, 2], tree.limits[:, 2]), v)
    position = np.zeros(tree.nv)
    position[tree.joint_dofs] = q[tree.joint_q]
    v = np.where(tree.position_limited, np.clip(v, (tree.limits[:, 0] - position) / h, (tree.limits[:, 1] - position) / h), v)
    return v, new


def exact_rollout(source, q, v, actions, friction, quality=False):
    """Observations [steps, envs, nq + nv] of an advance, in 64 bits."""

    tree = Tree(nb.world.compile_model(source, MODEL_SEED))
    contact = source == "tree29"
    substeps = SUBSTEPS if contact else 1
    h = float(np.float32(CONTROL_DT if contact else CHAIN_DT)) / substeps
    q, v = q.astype(np.float64), v.astype(np.float64)
    manifolds = [{} for _ in range(q.shape[0])]
    out = []
    for action in actions.astype(np.float64):
        target = np.zeros_like(v)
        target[:, tree.actuated] = action
        for _ in range(substeps):
            vf, H, kin = tree.dynamics(q, v, tree.drives(q, v, target, h), h)
            if contact:
                for e in range(q.shape[0]):
                    v[e], manifolds[e] = contact_substep(tree, q[e], v[e], vf[e], H[e], [k[e] for k in kin], manifolds[e],
                                                         float(friction[e]), h, quality)
            else:
                v = vf
            q = tree.integrate(q, v, h)
        out.append(np.concatenate([q, v], 1))
    return np.array(out)


def exact(case: dict, seed: int):
    """`run`'s floating outputs in 64 bits.  Piles have none: their all-pairs
    box, capsule, cylinder and hull queries would take a plain restatement
    minutes.  The task layer's frames and draws have none either."""

    envs, steps, kind = case["envs"], case["steps"], case["kind"]

    def rollout(source, n, quality=False):
        if source == "tree29" and n * steps > (EXACT_TREE_ENV_STEPS if not quality else 16):
            return None
        inputs = (tree_inputs if source == "tree29" else chain_inputs)(n, steps, seed)
        return exact_rollout(source, *inputs, nb.sample_reset(source, MODEL_SEED, seed, 0, n)[2], quality)

    if kind in ("scene", "policy"):
        return None
    if kind == "mix":
        n_chain, n_tree, n_pile = mix_counts(envs)
        parts = [rollout("chain7", n_chain), rollout("tree29", n_tree)]
        ends = [[None, None] if x is None else [x[-1, :, :nq], x[-1, :, nq:]] for x, nq in zip(parts, (7, 36))]
        return {"status": None, "state": ends + [[None, None]] * len(n_pile)}
    observations = rollout("chain7" if kind == "chain" else "tree29", envs, kind == "quality")
    if observations is None:
        return None
    if kind == "tree_host":
        return {"observations": observations, "status": None, "contacts": None, "final_q": observations[-1, :, :36]}
    return {"observations": observations, "status": None}
