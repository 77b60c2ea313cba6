"""Workloads of the batched step whose time is worth watching, through the public Python interface.

Four ways in which programs drive a world:

    policy   an RL loop: ``NukaVecEnv.step(actions)``, decimation 4, autoreset, the observation record
    host     a control loop on host arrays: ``upload`` the drive targets, step, ``download`` the robot state
    stream   a control loop on the GPU: commands are written into the world's own buffers, then ``step_n``
    rollout  sampling-based planning and data generation: reset, load start states, write commands, ``step_n`` a horizon

on the scenes of ``nuka.templates``.  Start states are mid-motion (feet and boxes about to touch or just touching, joints
and bases moving), commands are redrawn for every pass from a ring of eight, so that the solver meets live contacts rather
than robots that have come to rest.
"""
import functools
import math
import os
import sys
import weakref

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "nuka-physics_b200"))
import nuka  # noqa: E402
from nuka import Field as F, templates as T  # noqa: E402
from nuka.vec_env import NukaVecEnv  # noqa: E402

RING = 8                    # distinct command sets a caller cycles through
PD, TORQUE, VELOCITY, COMPUTED_TORQUE, OPERATIONAL_SPACE, ACTUATOR = 0, 1, 2, 3, 4, 5       # control modes of the world


def listed():
    def case(name, scene, call, envs, steps, control=PD, boxes=0, graph=False):
        return {"name": name, "scene": scene, "call": call, "envs": envs, "steps": steps, "control": control, "boxes": boxes, "graph": graph}

    return [
        # one robot under a trained policy (evaluation, a viewer, hardware-in-the-loop): all latency
        case("quadruped-policy-1", "quadruped", "policy", 1, 4),
        # a handful of robots driven from numpy, one physics step per control step
        case("quadruped-host-16", "quadruped", "host", 16, 1),
        # a batch that is no multiple of anything: a workstation-sized training run
        case("quadruped-policy-1000", "quadruped", "policy", 1000, 4),
        # the standard locomotion training batch
        case("quadruped-policy-4096", "quadruped", "policy", 4096, 4),
        # the same batch driven from host arrays with the robot state read back every step
        case("quadruped-host-4096", "quadruped", "host", 4096, 1),
        # the largest locomotion batch of one GPU
        case("quadruped-policy-16384", "quadruped", "policy", 16384, 4),
        # motor-model planning: open-loop efforts inside the torque-speed envelope over a short horizon
        case("quadruped-rollout-actuator-2500", "quadruped", "rollout", 2500, 10, ACTUATOR),
        # locomotion among loose objects
        case("quadruped-boxes-policy-4096", "quadruped", "policy", 4096, 4, boxes=4),
        # whole-body humanoid training with limb self-contact
        case("humanoid-policy-2048", "humanoid", "policy", 2048, 4),
        # manipulator planning without contacts: sampled joint targets over a horizon
        case("arm-rollout-4096", "arm7", "rollout", 4096, 32),
        # manipulators tracking a moving tool target in operational space
        case("arm-osc-1024", "arm7", "stream", 1024, 4, OPERATIONAL_SPACE),
        # clutter: stacked boxes that settle and topple, as grasp and packing data sets generate them
        case("pile48-rollout-1024", "pile", "rollout", 1024, 2, boxes=48),
    ]


def draw(rng):
    def count(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    scene = rng.choice(["quadruped"] * 5 + ["boxes"] * 2 + ["humanoid"] * 2 + ["arm7"] * 2 + ["pile"] * 2)
    case = {"scene": scene, "call": "policy", "envs": 1, "steps": 4, "control": PD, "boxes": 0, "graph": False}
    if scene == "quadruped":
        case["call"] = rng.choice(["policy", "policy", "host", "rollout"])
        if case["call"] == "policy":
            case.update(envs=count(1, 16384), steps=rng.choice([2, 4, 4, 5]))
        elif case["call"] == "host":
            case.update(envs=count(1, 8192), steps=rng.choice([1, 1, 2, 4]), graph=rng.choice([False, False, True]))
        else:
            case.update(envs=count(16, 4096), steps=rng.randint(4, 12), control=rng.choice([PD, TORQUE, VELOCITY, ACTUATOR]))
    elif scene == "boxes":
        case.update(scene="quadruped", boxes=rng.randint(1, 6), envs=count(1, 4096))
    elif scene == "humanoid":
        case.update(envs=count(1, 2048))
    elif scene == "arm7":
        if rng.random() < 0.5:
            case.update(call="rollout", envs=count(16, 8192), steps=rng.randint(8, 48), control=rng.choice([PD, TORQUE]))
        else:
            case.update(call="stream", envs=count(1, 4096), steps=rng.randint(1, 8), control=rng.choice([COMPUTED_TORQUE, OPERATIONAL_SPACE]),
                        graph=rng.choice([False, False, True]))
    else:
        case.update(call="rollout", boxes=rng.randint(6, 48), envs=count(1, 1024), steps=rng.randint(1, 2))
    return case


# ---- what a program has in hand before its loop ----------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def device():
    return nuka.Device.create(0, cuda_stream=stream().cuda_stream)


@functools.lru_cache(maxsize=None)
def stream():
    return torch.cuda.Stream()


@functools.lru_cache(maxsize=None)
def template(scene, boxes):
    if scene == "arm7":
        return T.arm7(0)
    if scene == "humanoid":
        return T.humanoid(0)
    if scene == "pile":
        return T.box_pile(0, count=boxes)
    return T.quadruped(0, boxes=boxes)


@functools.lru_cache(maxsize=None)
def cooked(scene, boxes):
    tb = template(scene, boxes)
    return tb.blob(), tb.arrays()


def release_with(world):
    """Gives the world's device memory back once neither the world nor a view of its buffers is held."""
    weakref.finalize(world, nuka._abi.lib().nuka_world_destroy, world._h)


def quaternions(turn):
    """Unit quaternions (wxyz) of small rotation vectors."""
    q = torch.cat([torch.ones_like(turn[..., :1]), 0.5 * turn], -1)
    return q / q.norm(dim=-1, keepdim=True)


def start_state(scene, boxes, envs, normal, uniform):
    """Per-env start state as {field: E x words float32}, and the joint positions the commands are drawn around."""
    arrays = cooked(scene, boxes)[1]
    links, rest = int(arrays["cfg_u"][4]), torch.from_numpy(arrays["q0"]).cuda()
    state = {}
    if scene == "pile":
        # columns of boxes on a 4 x 4 grid, each box turned and tilted and its centre half a millimetre too low to rest flat
        half = torch.from_numpy(arrays["shape_params"].reshape(-1, 4)[:boxes, :3]).cuda()
        pose = torch.zeros(envs, boxes + 1, 7, device="cuda")
        pose[..., 3] = 1.0
        top = torch.zeros(envs, 16, device="cuda")
        for k in range(boxes):
            column = k % 16
            pose[:, k, 0] = 0.25 * (column % 4 - 1.5) + 0.01 * normal(envs)
            pose[:, k, 1] = 0.25 * (column // 4 - 1.5) + 0.01 * normal(envs)
            pose[:, k, 2] = top[:, column] + half[k, 2] - 0.0005
            top[:, column] += 2.0 * half[k, 2] - 0.0005
            pose[:, k, 3:] = quaternions(torch.stack([0.08 * normal(envs), 0.08 * normal(envs), 0.3 * normal(envs)], 1))
        state[F.RIGID_BODY_TRANSFORM] = pose
        for field in (F.BODY_LINEAR_VELOCITY, F.BODY_ANGULAR_VELOCITY):
            velocity = torch.zeros(envs, boxes + 1, 3, device="cuda")
            velocity[:, :boxes] = 0.1 * normal(envs, boxes, 3)
            state[field] = velocity
        return state, rest
    q, qdot = torch.zeros(envs, links, device="cuda"), torch.zeros(envs, links, device="cuda")
    spread = {"arm7": 0.4, "humanoid": 0.1, "quadruped": 0.15}[scene]
    q[:, 1:] = rest[1:] + spread * normal(envs, links - 1)
    qdot[:, 1:] = 0.5 * normal(envs, links - 1)
    state[F.JOINT_POSITION], state[F.JOINT_VELOCITY] = q, qdot
    if scene == "arm7":
        return state, rest
    base = torch.from_numpy(arrays["base_pose0"]).cuda().repeat(envs, 1)
    base[:, 3:] = quaternions(0.03 * normal(envs, 3))
    if scene == "quadruped":
        # the lowest foot sphere just inside the ground: hip roll, thigh and shank of 0.213 m, foot radius 0.022 m
        roll, thigh, shank = (q[:, 1:].reshape(envs, 4, 3)[..., k] for k in range(3))
        side = torch.tensor([0.08, -0.08, 0.08, -0.08], device="cuda")
        foot = side * torch.sin(roll) - 0.213 * (torch.cos(thigh) + torch.cos(thigh + shank)) * torch.cos(roll)
        base[:, 2] = 0.022 - foot.min(1).values + uniform(envs, -0.002, 0.004)
    else:
        base[:, 2] += uniform(envs, -0.006, 0.01)
    state[F.BASE_POSE] = base
    twist = torch.zeros(envs, links, 6, device="cuda")
    twist[:, 0] = 0.2 * normal(envs, 6)
    state[F.LINK_VELOCITY] = twist
    if boxes:
        pose = torch.from_numpy(arrays["body_pose0"]).cuda().reshape(1, -1, 7).repeat(envs, 1, 1)
        free = torch.from_numpy(arrays["inv_mass"] > 0.0).cuda()
        pose[:, free, :2] += 0.05 * normal(envs, boxes, 2)
        pose[:, free, 2] += 0.001 * normal(envs, boxes)
        pose[:, free, 3:] = quaternions(torch.cat([0.05 * normal(envs, boxes, 2), normal(envs, boxes, 1)], -1))
        state[F.RIGID_BODY_TRANSFORM] = pose
    return state, rest


def commands(scene, control, envs, links, rest, q, normal):
    """One command set: {field: E x words}."""
    noise = torch.zeros(envs, links, device="cuda")
    noise[:, 1:] = normal(envs, links - 1)
    if control == TORQUE or control == ACTUATOR:
        return {F.DRIVE_TARGET: 2.0 * noise}
    if control == VELOCITY:
        return {F.VELOCITY_TARGET: noise}
    if control == OPERATIONAL_SPACE:
        tip = torch.tensor([1.2, 0.0, 0.9], device="cuda")           # in front of the stretched arm
        return {F.TASK_TARGET: tip + 0.1 * normal(envs, 3)}
    target = {F.DRIVE_TARGET: (q if scene == "arm7" else rest) + 0.15 * noise}
    if control == COMPUTED_TORQUE:
        target[F.VELOCITY_TARGET] = 0.5 * noise
        target[F.ACCELERATION_TARGET] = 2.0 * noise
    return target


def gains(scene, control, envs, links):
    def every(value):
        return torch.full((envs, links), value, device="cuda")

    if scene == "arm7":
        if control == PD:
            return {F.DRIVE_STIFFNESS: every(60.0), F.DRIVE_DAMPING: every(4.0)}
        if control == COMPUTED_TORQUE:
            return {F.DRIVE_STIFFNESS: every(25.0), F.DRIVE_DAMPING: every(3.0)}
        if control == OPERATIONAL_SPACE:
            kp, kd = torch.zeros(envs, links, device="cuda"), torch.zeros(envs, links, device="cuda")
            kp[:, 7], kd[:, 7] = 25.0, 10.0
            frame = torch.tensor([0.3, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0], device="cuda").repeat(envs, 1)
            posture = torch.full((envs, 1), 20.0, device="cuda")
            return {F.DRIVE_STIFFNESS: kp, F.DRIVE_DAMPING: kd, F.TASK_LOCAL_POSE: frame, F.TASK_NULLSPACE_STIFFNESS: posture,
                    F.TASK_NULLSPACE_DAMPING: posture}
        return {}
    if control == VELOCITY:
        return {F.DRIVE_STIFFNESS: every(8.0), F.DRIVE_FORCE_LIMIT: every(15.0)}
    if control == ACTUATOR:
        return {F.DRIVE_FORCE_LIMIT: every(3.0), F.ACTUATOR_NOLOAD_SPEED: every(6.0)}
    return {}


class State:
    """What the caller's loop holds: the world (or the vectorised env), command ring, start state, views to read."""


def prepare(case, seed):
    with torch.cuda.stream(stream()):            # the world's stream: what follows is ordered behind the world's own set-up
        s = build(case, torch.Generator(device="cuda").manual_seed(seed))
    s.world.synchronize()
    return s


def build(case, gen):
    scene, boxes, envs, control = case["scene"], case["boxes"], case["envs"], case["control"]

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    def uniform(n, lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=gen, device="cuda")

    blob, arrays = cooked(scene, boxes)
    links = int(arrays["cfg_u"][4])
    s = State()
    s.call, s.steps, s.turn = case["call"], case["steps"], 0
    start, rest = start_state(scene, boxes, envs, normal, uniform)
    if s.call == "policy":
        s.env = NukaVecEnv(device(), blob, envs, decimation=s.steps)
        s.world = s.env.world
        release_with(s.world)
        s.env.reset()
        # episodes are out of phase, as after a learner's first iterations
        s.env.episode_steps.random_(0, s.env.max_episode_length, generator=gen)
        s.ring = [0.6 * normal(envs, links - 1) for _ in range(RING)]
    else:
        osc = {"osc_task_link": links - 1} if control == OPERATIONAL_SPACE else {}
        s.world = nuka.World.create_from_template(device(), blob, envs, control_mode=control, **osc)
        release_with(s.world)
        s.world.set_execution_mode(case["graph"])
        for field, value in gains(scene, control, envs, links).items():
            s.world.view(field).torch().copy_(value)
        s.ring = [commands(scene, control, envs, links, rest, start.get(F.JOINT_POSITION), normal) if links else {} for _ in range(RING)]
        if s.call == "host":
            s.ring = [{field: value.cpu().numpy() for field, value in c.items()} for c in s.ring]
        else:
            s.views = {field: s.world.view(field).torch() for field in s.ring[0]}
    s.start = [(s.world.view(field).torch(), value.reshape(envs, -1)) for field, value in start.items()]
    for view, value in s.start:
        view.copy_(value)
    s.world.forward_kinematics()
    fields = [F.JOINT_POSITION, F.JOINT_VELOCITY, F.ARTICULATION_LINK_POSE, F.LINK_VELOCITY, F.ACTUATOR_EFFORT] if links else []
    if boxes:
        fields += [F.RIGID_BODY_TRANSFORM, F.BODY_LINEAR_VELOCITY, F.BODY_ANGULAR_VELOCITY]
    s.out = {field.name: s.world.view(field).torch() for field in fields}
    return s


def run(s):
    command = s.ring[s.turn % RING]
    s.turn += 1
    if s.call == "policy":
        obs, reward, terminated, truncated, _ = s.env.step(command)
        return {"obs": obs, "reward": reward, "terminated": terminated, "truncated": truncated, **s.out}
    if s.call == "host":
        for field, value in command.items():
            s.world.upload(field, value)
        s.world.step_n(s.steps)
        return [s.world.download(field) for field in (F.JOINT_POSITION, F.JOINT_VELOCITY, F.BASE_POSE, F.LINK_VELOCITY)]
    with torch.cuda.stream(stream()):
        if s.call == "rollout":
            s.world.reset()
            for view, value in s.start:
                view.copy_(value)
            s.world.forward_kinematics()
        for field, view in s.views.items():
            view.copy_(command[field])
        s.world.step_n(s.steps)
    return s.out


def work(case):
    """Each input array read once and each output array written once per pass; operations of one kinematics, mass-matrix,
    narrowphase and single-Newton-step pass per env-step (the solver's sweeps beyond the first are not counted)."""
    arrays = cooked(case["scene"], case["boxes"])[1]
    links, free = int(arrays["cfg_u"][4]), case["boxes"]
    dofs = T.dof_count(arrays)
    floating = dofs > 7
    points = {"arm7": 0, "quadruped": 4, "humanoid": 8, "pile": 0}[case["scene"]] + 4 * free
    # in: q, qdot, six drive inputs, base pose and twist, carried velocities, bodies, cached points; out: coordinates, efforts,
    # poses, twists, the same carried state, contact read-outs
    words = 8 * links + 13 * floating + dofs + 19 * free + 10 * points
    words += 5 * links + 13 * links + 7 * floating + dofs + 19 * free + 18 * points
    if case["call"] == "policy":
        words += 2 * (links - 1) + 12 + 3 * (links - 1) + 3
    elif case["call"] == "rollout":
        words += 2 * links + 13 * floating + 13 * free
    flops = 900 * links + dofs ** 3 // 3 + 4 * dofs ** 2                                   # kinematics, bias, inertia; factor and solve
    flops += dofs ** 3 // 3 + 6 * dofs ** 2 + min(points, 8) * 6 * dofs * dofs if links else 0   # one Newton step of the articulation
    flops += free * (600 + 4 * 300) + points * 150                                         # rigid blocks, manifolds and rows
    return {"bytes": 4 * words * case["envs"], "flops": flops * case["envs"] * case["steps"]}


def tolerance(case):
    """Relative differences between two evaluations in 32-bit floats that round differently (fused or separate multiply-adds),
    with room for the worst env of a batch.  A pass is several steps, each an iterative contact solve that stops at an
    absolute residual or a sweep limit, so last-bit differences grow; a box on a box also picks its separating axis and its
    four contact points by comparisons that such a difference can turn."""
    if case["scene"] == "pile":
        return {"rel": 1e-2, "max": 0.9}
    if case["boxes"]:
        return {"rel": 3e-3, "max": 0.5, "differ": 0.002}
    if case["scene"] == "arm7":
        return {"rel": 5e-5, "max": 1e-3}
    if case["call"] == "rollout":
        return {"rel": 1e-3, "max": 0.1}
    return {"rel": 1e-4, "max": 2e-2, "differ": 0.002}
