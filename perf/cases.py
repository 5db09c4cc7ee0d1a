"""Timed workloads of the simulator: what a program that uses this framework has it do.

Every case is one pass through the public entry points -- the batch front-end
(``MassSpringBatch``), the gym client, the MPM batch, the library's own
admission / poll loop and the no-allocation call -- on seeded synthetic robots.
The robots are those of the repository's configurations: the quadruped lattice
(93 vertices, MLP 1x64), the spider lattice (236 vertices, MLP 2x256), random
lattices of 50-2000 vertices with a controller each (MLP 2x128), the
reference's cube robots with its own controller layout and losses, and the
legged MPM body on a 64^3 grid.  Physics is the synthetic configurations'
(``workloads.PHYSICS``).  Episodes are windows of those configurations'
episodes, short enough that single precision still determines their gradients
(they lose that over thousands of contact-rich substeps); the loss windows open
early (``run_period``), as they are open for nearly all of a long episode.

Kinds of case:

* ``gym``     an external policy drives the robot step by step (reinforcement
              learning, ``clients.MassSpringEnvCUDA``): latency of one call.
* ``eval``    forward-only rollout of trained controllers, observables and
              final state read back.
* ``train``   one training iteration: rollout, loss, reverse pass and the
              optimiser step; gradients stay on the device.
* ``serve``   rollout and gradient requests of mixed lengths admitted to a pool
              of slots and polled to completion.
* ``mpm``     MLS-MPM rollout, with the reverse pass or without it.
* ``advance`` mass-spring substeps on the caller's own device buffers.

``exact`` restates the simulation in 64-bit torch with autograd.
"""
import ctypes
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import cls_b200
from cls_b200 import clients, mpm, robot_design, sharding, workloads
from cls_b200.batch import MassSpringBatch, Robot

LIFT = np.array([0.0, 0.1, 0.0])
ACT_SCALE = 0.2          # the controller sees (x - centre) / 0.2
# Losses of the single-precision training cases.  A robot with a controller of its
# own trains on its posture here: the velocity loss pushes all its vertices alike,
# a thousand times harder than the rotation loss does, and of such a push only the
# rounding reaches its controller until it lands.
FP32_LOSSES = ("velocity", "rotation")
OWN_LOSSES = ("rotation",)
ALL_LOSSES = ("velocity", "height", "pose", "actuation", "rotation", "crawl")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a policy in training steps one robot: 16 calls, each an observation
        dict(name="gym_quadruped_1", kind="gym", robot="quadruped", envs=1, steps=16),
        # a trained controller shown on one robot: the smallest whole rollout
        dict(name="eval_quadruped_1", kind="eval", robot="quadruped", envs=1, steps=100),
        # the plain configuration: 32 envs share a 1x64 controller, one segment
        dict(name="train_quadruped_32", kind="train", robot="quadruped", envs=32, steps=100, every=100, adam=True),
        # the reference's own setting in double precision: sine controller with
        # an output per spring, duplicated goal inputs, every loss, odd batch
        dict(name="train_cubes_fp64", kind="train", robot="cubes", envs=7, steps=113, every=25, precision=64),
        # the large batch: 4096 envs share a 2x256 controller
        dict(name="train_spider_4096", kind="train", robot="spider", envs=4096, steps=80, every=80),
        # a ragged mid-size batch over several segments, replayed as a graph
        dict(name="train_spider_300", kind="train", robot="spider", envs=300, steps=90, every=40, graph=True),
        # a few robots of very different sizes, fewer than the GPU has SMs
        dict(name="train_lattices_24", kind="train", robot="lattices", robots=24, vmin=50, vmax=2000, shape=5,
             steps=91, every=25),
        # the uneven batch: 512 robots, each its own controller, checkpoints every 50
        dict(name="train_lattices_512", kind="train", robot="lattices", robots=512, vmin=50, vmax=2000, shape=0,
             steps=121, every=50),
        # requests of mixed lengths, a third with gradients, on 16 slots
        dict(name="serve_16", kind="serve", slots=16, requests=28, vertices=300, shape=3, max_steps=120, every=20),
        # the MPM configuration: 8 envs of the legged body, forward and reverse
        dict(name="mpm_body_8", kind="mpm", dim=3, envs=8, steps=75, every=50, grad=True),
        # the reference's 2D solver constants on a small body
        dict(name="mpm_square_2", kind="mpm", dim=2, envs=2, steps=120, every=50, side=10, grad=True),
        # a host runtime that owns its memory advances 64 quadrupeds
        dict(name="advance_64", kind="advance", robot="quadruped", envs=64, steps=32),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gym", "eval", "train", "train", "train", "serve", "mpm", "advance"])
    if kind == "gym":
        return dict(kind=kind, robot=rng.choice(["quadruped", "spider"]), envs=_spread(rng, 1, 48), steps=rng.randint(6, 24))
    if kind == "eval":
        return dict(kind=kind, robot=rng.choice(["quadruped", "spider"]), envs=_spread(rng, 1, 200),
                    steps=rng.randint(50, 100))
    if kind == "serve":
        return dict(kind=kind, slots=2 * rng.randint(3, 10), requests=rng.randint(12, 36), vertices=_spread(rng, 150, 900),
                    shape=rng.randint(0, 999), max_steps=rng.randint(60, 130), every=rng.randint(10, 50))
    if kind == "mpm":
        if rng.random() < 0.4:
            return dict(kind=kind, dim=2, envs=_spread(rng, 1, 16), steps=rng.randint(40, 150), every=rng.randint(20, 60),
                        side=rng.randint(6, 16), grad=rng.random() < 0.6)
        return dict(kind=kind, dim=3, envs=rng.randint(1, 8), steps=rng.randint(20, 75), every=rng.randint(20, 60),
                    grad=rng.random() < 0.6)
    if kind == "advance":
        return dict(kind=kind, robot=rng.choice(["quadruped", "spider"]), envs=_spread(rng, 1, 1000), steps=rng.randint(8, 64))
    robot = rng.choice(["quadruped", "spider", "lattices", "lattices", "cubes"])
    steps = rng.randint(50, 100)
    if robot == "lattices":
        vmax = _spread(rng, 120, 2000)
        return dict(kind=kind, robot=robot, robots=_spread(rng, 1, 300), vmin=50, vmax=vmax, shape=rng.randint(0, 999),
                    steps=steps, every=rng.randint(20, 50))
    if robot == "cubes":
        return dict(kind=kind, robot=robot, envs=_spread(rng, 1, 24), steps=steps, every=rng.randint(15, 60),
                    precision=rng.choice([32, 64]))
    return dict(kind=kind, robot=robot, envs=_spread(rng, 1, 3000 if robot == "spider" else 1000), steps=steps,
                every=rng.choice([steps, rng.randint(20, 50)]), adam=rng.random() < 0.5)


# ------------------------------------------------------- robots and parameters
@functools.lru_cache(maxsize=64)
def _lattices(n, vmin, vmax, shape):
    return tuple(workloads.uneven_robots(n, seed=shape, vmin=vmin, vmax=vmax))


@functools.lru_cache(maxsize=None)
def _robot(name):
    if name == "quadruped":
        return Robot.actuated_outputs(*robot_design.quadruped_lattice(), hidden=[64])
    if name == "spider":
        return Robot.actuated_outputs(*robot_design.spider_lattice(), hidden=[256, 256])
    objects, springs = robot_design.reference_robot(101, 3e4, 0.2)
    return Robot(objects, springs, hidden=[32])


def _robots(case):
    """(robot types, envs of each): the random lattices are one env each."""
    if case["robot"] == "lattices":
        return list(_lattices(case["robots"], case["vmin"], case["vmax"], case["shape"])), 1
    return [_robot(case["robot"])], case["envs"]


def _params(case, T, steps):
    """Keyword arguments of ``default_params`` for a mass-spring case."""
    every = case.get("every", 50)
    if case.get("robot") == "cubes":     # the reference's schema: its own controller input and losses
        p = dict(dt=4e-3, gravity=-1.8, ground_height=0.1, friction=0.4, drag_damping=0.0, dashpot_damping=0.1,
                 stiffness_scale=0.1, max_steps=T, checkpoint_every=every, run_period=20, turn_period=50, jump_period=25,
                 spring_omega=2 * math.pi / 4e-3 / 100, n_sin_waves=10, duplicate_v=5, duplicate_h=3, duplicate_c=2,
                 activation_hidden="sin", activation_output="sin", loss=list(ALL_LOSSES), max_speed=0.1, max_height=0.1)
    else:
        own = case["kind"] == "serve" or case.get("robot") == "lattices"
        p = workloads._params(T, every, run_period=30, loss=OWN_LOSSES if own else FP32_LOSSES)
    p["precision"] = case.get("precision", 32)
    return p


def _state(robots, envs, seed, lift=0.0, turned=False):
    """Initial positions and velocities, env after env: the rest poses with
    noise, `turned` to a heading drawn from the seed."""
    g = np.random.default_rng(seed)
    objects = np.concatenate([np.tile(r.objects, (envs, 1)) for r in robots])
    if turned:
        a = np.random.default_rng(seed + 4).uniform(0.2, 0.8)
        objects = objects @ np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]])
    return objects + g.uniform(-2e-3, 2e-3, objects.shape) + lift, g.uniform(-0.05, 0.05, objects.shape)


def _lift(case):
    """Large training batches in single precision are dropped from 10 cm: which of
    two neighbouring substeps a vertex lands in is a rounding decision, and among
    thousands of landings one that falls the other way moves the batch's
    gradient by 1e-4.  The other cases land, or stand on the ground throughout."""
    large = case.get("robot") == "lattices" or case["envs"] > 64
    return LIFT if case["kind"] == "train" and large else 0.0


def _targets(case, T, n_envs, seed):
    g = np.random.default_rng(seed + 1)
    if case.get("robot") == "cubes":     # goals that open every loss term for some env
        tv, th, tc = np.zeros((T, n_envs, 3)), np.zeros((T, n_envs)), np.zeros((T, n_envs))
        tv[:, :, 0], tv[:, :, 2] = g.uniform(-0.1, 0.1, n_envs), g.uniform(-0.1, 0.1, n_envs)
        th[:] = g.uniform(0.0, 0.3, n_envs)
        tc[:] = np.arange(n_envs) % 2
        return tv, th, tc
    tv, th = workloads.targets(g, T, n_envs)
    return tv, th, np.zeros((T, n_envs))


def _cast(case, a):
    """A single-precision handle's values, which the C interface hands out as
    doubles, in the type they were computed in."""
    return np.asarray(a, np.float64 if case.get("precision", 32) == 64 else np.float32)


def _batch(case, T, steps, seed):
    robots, envs = _robots(case)
    b = MassSpringBatch(robots, [r for r in range(len(robots)) for _ in range(envs)],
                        cls_b200.default_params(**_params(case, T, steps)))
    b.weights_init(seed + 2)
    b.set_targets(*_targets(case, T, b.n_envs, seed))
    b.set_state(*_state(robots, envs, seed, _lift(case), case["kind"] == "eval"))
    return b


# -------------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](dict(case), int(seed))


def run(state):
    return state["run"](state)


def _prepare_gym(case, seed):
    robot, steps = _robot(case["robot"]), case["steps"]
    T = steps + 2
    env = clients.MassSpringEnvCUDA(robot, case["envs"], cls_b200.default_params(**_params(case, T, steps)), seed=seed,
                                    training=False, initial_objects=_state([robot], 1, seed)[0])
    return dict(case=case, run=_run_gym, env=env, actions=_actions(case, seed))


def _actions(case, seed):
    n = int((_robot(case["robot"]).springs[:, 4] > 0).sum())
    return np.random.default_rng(seed + 3).uniform(-1, 1, (case["steps"], case["envs"], n))


def _run_gym(s):
    env, obs, rewards = s["env"], [], []
    obs.append(env.reset())
    for a in s["actions"]:
        o, r, _, _ = env.step(a)
        obs.append(o)
        rewards.append(r)
    return dict(obs=_cast(s["case"], np.stack(obs)), reward=_cast(s["case"], rewards))


def _prepare_eval(case, seed):
    return dict(case=case, run=_run_eval, batch=_batch(case, case["steps"] + 2, case["steps"], seed))


def _run_eval(s):
    b = s["batch"]
    b.forward_eval(s["case"]["steps"])
    out = b.observables()
    out["x"], out["v"] = b.final_state()
    return {k: _cast(s["case"], v) for k, v in out.items()}


def _prepare_train(case, seed):
    b = _batch(case, case["steps"], case["steps"], seed)
    stream = None
    if case.get("graph"):
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        b.graph_capture(case["steps"], with_adam=True)
    return dict(case=case, run=_run_train, batch=b, stream=stream, it=0)


def _run_train(s):
    b, case = s["batch"], s["case"]
    if case.get("graph"):
        b.graph_launch(s["it"])
        env = b.loss()[1]
    else:
        b.forward(case["steps"])
        env = b.loss()[1]
        b.backward()
        if case.get("adam"):
            b.adam_step(s["it"])
    s["it"] += 1
    grads = sharding.grad_tensors(b)
    for g in grads:
        g.batch = b        # views of the batch's own buffers: they live as long as it does
    return dict(loss=_cast(case, env), grads=grads)


# A pool of slots: half for a lattice of 100 vertices, half for a larger one; the
# slots of a class hold the same controller, as a deployed one would be.
def _serve_robots(case):
    return [_lattices(1, n, n, case["shape"])[0] for n in (100, case["vertices"])]


def _serve_requests(case, seed):
    g, mix = np.random.default_rng(seed + 5), np.random.default_rng(case["shape"])   # the mix is the case's own
    out = []
    for k in range(case["requests"]):
        kind = int(mix.integers(2))
        robot = _serve_robots(case)[kind]
        T = case["max_steps"]
        tv = np.zeros((T, 3))
        tv[:, 0], tv[:, 2] = g.uniform(-0.1, 0.1), g.uniform(-0.1, 0.1)
        out.append(dict(kind=kind, steps=int(mix.integers(min(40, T // 2), T + 1)), grad=k % 3 == 0,
                        x0=robot.objects + g.uniform(-2e-3, 2e-3, robot.objects.shape) + LIFT,
                        tv=tv, th=np.full(T, g.uniform(-0.1, 0.1))))
    return out


def _serve_weights(case, seed):
    """[kind][layer] (W, b) in the reference layout."""
    g = np.random.default_rng(seed + 6)
    out = []
    for r in _serve_robots(case):
        widths = [8 + 6 * r.n_vertices + 3] + list(r.hidden) + [r.n_outputs]
        out.append([(g.uniform(-1, 1, (o, i)) * math.sqrt(6.0 / i), g.uniform(-0.1, 0.1, o))
                    for i, o in zip(widths, widths[1:])])
    return out


def _prepare_serve(case, seed):
    half = case["slots"] // 2
    robots = [r for r in _serve_robots(case) for _ in range(half)]
    p = cls_b200.default_params(**_params(case, case["max_steps"], case["max_steps"]))
    b = MassSpringBatch(robots, list(range(len(robots))), p)
    for slot in range(len(robots)):
        for layer, (W, bias) in enumerate(_serve_weights(case, seed)[slot // half]):
            b.set_weights(slot, layer, W, bias)
    b.serve_tick(1)
    return dict(case=case, run=_run_serve, batch=b, half=half, requests=_serve_requests(case, seed))


def _run_serve(s):
    b, reqs, half = s["batch"], s["requests"], s["half"]
    waiting, n = list(range(len(reqs))), len(reqs)
    done, losses, final, grads = 0, [None] * n, [None] * n, [None] * n
    while done < n:
        left = []
        for k in waiting:
            r = reqs[k]
            slot = b.admit(k + 1, r["kind"] * half, r["steps"], grad=r["grad"], x0=r["x0"], target_v=r["tv"],
                           target_h=r["th"])
            if slot < 0:
                left.append(k)
        waiting = left
        ids, _ = b.poll()
        for rid in ids:
            k = rid - 1
            slot, losses[k], final[k] = b.serve_result(rid)
            if reqs[k]["grad"]:
                grads[k] = np.concatenate([a.ravel() for l in range(b.n_layers(slot)) for a in b.get_grads(slot, l)])
            b.serve_release(rid)
            done += 1
    case = s["case"]
    return dict(loss=_cast(case, np.stack(losses)), x=_cast(case, np.concatenate([f.ravel() for f in final])),
                grad=_cast(case, np.concatenate([g for g in grads if g is not None])))


def _mpm_body(case):
    """positions, muscle, fibre (None: the vertical default), number of muscles and solver parameters."""
    if case["dim"] == 3:
        pos, mus, fib = workloads.legged_body(n_grid=64)
        E, nu = 1e4, 0.3
        return pos, mus, fib, 16, dict(n_grid=64, bound=3, material="neo_hookean", dt=1e-4, gravity=-10.0, p_vol=1.0,
                                       mu=E / (2 * (1 + nu)), la=E * nu / ((1 + nu) * (1 - 2 * nu)), act_strength=1e3,
                                       mass=1.0)
    side, dx = case["side"], 1.0 / 32      # a square of side x side cells, 4 particles each, 4 muscles in its lower half
    i, j, a, b = np.meshgrid(np.arange(side), np.arange(side), (0.25, 0.75), (0.25, 0.75), indexing="ij")
    pos = np.stack([(5 + i + a).ravel() * dx, (4 + j + b).ravel() * dx], axis=1)
    mus = np.where(j.ravel() < side // 2, (i.ravel() * 4) // side, -1).astype(np.int32)
    return pos, mus, None, 4, dict(n_grid=32, bound=3, material="fixed_corotated", dt=1e-3, gravity=-10.0, p_vol=1.0,
                                   mu=40.0, la=40.0, act_strength=4.0, mass=1.0)


def _mpm_inputs(case, seed):
    """Initial state, muscle drive and loss of an MPM case."""
    pos, _, _, M, p = _mpm_body(case)
    g, T, E, D = np.random.default_rng(seed), case["steps"], case["envs"], case["dim"]
    x0 = np.broadcast_to(pos, (E,) + pos.shape).copy()
    v0 = np.broadcast_to(g.uniform(-0.3, 0.3, (E, 1, D)), x0.shape).copy()
    t = np.arange(T)[:, None, None] * p["dt"]
    act = np.sin(2 * np.pi * g.uniform(2.0, 6.0, (1, E, M)) * t + g.uniform(0, 2 * np.pi, (1, E, M)))
    w = np.zeros(T + 1)
    w[T] = 1.0
    target = np.broadcast_to(pos.mean(axis=0) + 0.05, (T + 1, E, D)).copy()
    return x0, v0, act, w, target


def _prepare_mpm(case, seed):
    pos, mus, fib, M, p = _mpm_body(case)
    x0, v0, act, w, target = _mpm_inputs(case, seed)
    b = mpm.MPMBatch(pos, mus, case["envs"], dim=case["dim"], fibre=fib, n_muscles=M, max_steps=case["steps"],
                     checkpoint_every=case["every"], precision=32, **p)
    b.set_state(x0, v0)
    b.set_actuation(act)
    b.set_loss(w, target)
    return dict(case=case, run=_run_mpm, batch=b)


def _run_mpm(s):
    b, case = s["batch"], s["case"]
    b.forward(case["steps"])
    loss = b.loss()
    if not case["grad"]:
        x, v, _, _ = b.final_state()
        return dict(loss=_cast(case, loss), centers=_cast(case, b.centers()), x=_cast(case, x), v=_cast(case, v))
    b.backward()
    act = np.zeros((b.T, b.E, b.M))       # what a muscle drive is trained with; initial-state gradients are not asked for
    b._c(b.lib.cls_mpm_get_grads(b.h, cls_b200._capi.ptr(act), None, None, None, None))
    return dict(loss=_cast(case, loss), centers=_cast(case, b.centers()), act=_cast(case, act))


class _Advance(ctypes.Structure):
    """cls_noalloc_advance of include/cls_b200.h."""
    _fields_ = ([(n, ctypes.c_int32) for n in ("n_envs", "n_vertices", "n_springs", "n_substeps")] +
                [(n, ctypes.c_void_p) for n in ("spring_a", "spring_b", "rest_length", "stiffness", "actuation_coef",
                                                "actuation", "x", "v")] +
                [(n, ctypes.c_float) for n in ("dt", "gravity", "ground_height", "drag_damping", "dashpot_damping",
                                               "friction")] +
                [("error_message", ctypes.c_char_p), ("error_capacity", ctypes.c_int32)])


def _advance_inputs(case, seed):
    robot, E = _robot(case["robot"]), case["envs"]
    x0, v0 = _state([robot], E, seed)
    act = np.random.default_rng(seed + 3).uniform(-1, 1, (E, robot.n_springs))
    return robot, x0.reshape(E, -1, 3), v0.reshape(E, -1, 3), act


def _prepare_advance(case, seed):
    robot, x0, v0, act = _advance_inputs(case, seed)
    dev = lambda a, t=torch.float32: torch.tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    sp, ph = robot.springs, workloads.PHYSICS
    t = dict(spring_a=dev(sp[:, 0], torch.int32), spring_b=dev(sp[:, 1], torch.int32), rest_length=dev(sp[:, 2]),
             stiffness=dev(sp[:, 3] * ph["stiffness_scale"]), actuation_coef=dev(sp[:, 4]), actuation=dev(act),
             x=dev(x0), v=dev(v0))
    args = _Advance(n_envs=case["envs"], n_vertices=robot.n_vertices, n_springs=robot.n_springs, n_substeps=case["steps"],
                    **{k: a.data_ptr() for k, a in t.items()}, dt=ph["dt"], gravity=ph["gravity"],
                    ground_height=ph["ground_height"], drag_damping=ph["drag_damping"],
                    dashpot_damping=ph["dashpot_damping"], friction=ph["friction"])
    fn = cls_b200._capi.load().cls_ms_advance_noalloc
    fn.argtypes, fn.restype = [ctypes.POINTER(_Advance), ctypes.c_void_p], ctypes.c_int32
    return dict(case=case, run=_run_advance, args=args, fn=fn, tensors=t)


def _run_advance(s):
    rc = s["fn"](ctypes.byref(s["args"]), torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError("cls_ms_advance_noalloc: %d" % rc)
    return dict(x=s["tensors"]["x"], v=s["tensors"]["v"])


# ----------------------------------------------------------------------- work
def _widths(case, r):
    p = _params(case, 2, 2)
    goals = 2 * (p["duplicate_v"] > 0) + (p["duplicate_h"] > 0) + (p["duplicate_c"] > 0)
    pos = -(-3 * r.n_vertices // 4) * 4
    return [pos + p["n_sin_waves"] + goals] + list(r.hidden) + [r.n_outputs or r.n_springs]


SPRING_FLOPS, SPRING_ADJ_FLOPS = 50, 110


def work(case):
    """Inputs read once, outputs written once; arithmetic of every substep."""
    kind, steps = case["kind"], case.get("steps", 0)
    if kind == "mpm":
        pos, _, _, M, p = _mpm_body(case)
        D, P = case["dim"], pos.shape[0] * case["envs"]
        per = (2 * 3 ** D) * (D * D + D + 1) * 2 * (3.0 if case["grad"] else 1.0)
        io = 4 * P * (2 * D + (0 if case["grad"] else 2 * D)) + 4 * steps * case["envs"] * (M * 2 + D)
        return dict(bytes=float(io), flops=per * P * steps)
    if kind == "serve":
        b = f = 0.0
        for r in _serve_requests(case, 0):
            robot = _serve_robots(case)[r["kind"]]
            w = _widths(case, robot)
            n = sum(i * o for i, o in zip(w, w[1:]))
            f += r["steps"] * ((2 * n + SPRING_FLOPS * robot.n_springs) +
                               (4 * n + SPRING_ADJ_FLOPS * robot.n_springs if r["grad"] else 0))
            b += 4 * (n * (2 if r["grad"] else 1) + 9 * robot.n_vertices)
        return dict(bytes=b, flops=f)
    if kind == "advance":
        r = _robot(case["robot"])
        return dict(bytes=4.0 * case["envs"] * (12 * r.n_vertices + r.n_springs) + 20.0 * r.n_springs,
                    flops=float(SPRING_FLOPS) * case["envs"] * r.n_springs * steps)
    robots, envs = _robots(case)
    size = 8 if case.get("precision", 32) == 64 else 4
    b = f = 0.0
    for r in robots:
        w = _widths(case, r)
        n = sum(i * o for i, o in zip(w, w[1:])) if kind != "gym" else 0
        passes = 2 if kind == "train" else 1
        b += size * (n * passes + envs * (6 * r.n_vertices * passes + 10 * r.n_springs / envs))
        f += envs * steps * (2 * n + SPRING_FLOPS * r.n_springs)
        if kind == "train":
            f += envs * steps * (4 * n + SPRING_ADJ_FLOPS * r.n_springs)
        if kind == "eval":
            b += size * envs * (6 * r.n_vertices + 6 * steps)
        if kind == "gym":
            b += size * envs * (steps + 1) * (w[0] + 3 * r.n_vertices + w[-1])
    return dict(bytes=float(b), flops=float(f))


# ---------------------------------------------------------------------- exact
def _t64(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _idx(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int64, device="cuda")


def _s64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _uniform(seed, stream, n):
    """The first n values of stream `stream` of the splitmix64 generator that
    weights_init documents (counter-based, 53 bits)."""
    gamma = 0x9E3779B97F4A7C15
    z = torch.arange(n, dtype=torch.int64, device="cuda") + _s64(seed * gamma + stream * 0xD1B54A32D192ED03 + gamma)
    shr = lambda a, k: (a >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
    z = (z ^ shr(z, 30)) * _s64(0xBF58476D1CE4E5B9)
    z = (z ^ shr(z, 27)) * _s64(0x94D049BB133111EB)
    return shr(z ^ shr(z, 31), 11).double() * 2.0 ** -53


class _Model:
    """Envs of several robot types as [V, E, ...] fields: the types' vertices,
    springs and outputs end to end, E envs of each."""

    def __init__(self, robots, envs, p):
        self.p, self.R, self.E = p, len(robots), envs
        self.robots = robots
        nv, self.nout = [r.n_vertices for r in robots], [r.n_outputs or r.n_springs for r in robots]
        voff, ooff = np.cumsum([0] + nv), np.cumsum([0] + self.nout)
        self.V, self.O = int(voff[-1]), int(ooff[-1])
        self.n = _t64(nv)[:, None, None]
        self.rob = _idx(np.repeat(np.arange(self.R), nv))
        sp = np.concatenate([r.springs for r in robots])
        off = np.repeat(voff[:-1], [r.n_springs for r in robots])
        self.sa, self.sb = _idx(sp[:, 0].astype(int) + off), _idx(sp[:, 1].astype(int) + off)
        self.len, self.coef = _t64(sp[:, 2])[:, None], _t64(sp[:, 4])[:, None]
        self.k = _t64(sp[:, 3])[:, None] * p["stiffness_scale"]
        self.ns = [r.n_springs for r in robots]
        out = [np.arange(r.n_springs) if r.spring_output is None else r.spring_output for r in robots]
        self.out = _idx(np.concatenate([np.where(o >= 0, o + a, self.O) for o, a in zip(out, ooff)]))
        # controller: layer widths padded to the largest robot's
        self.pos_pad = [-(-3 * n // 4) * 4 for n in nv]
        self.goals = [2 * (p["duplicate_v"] > 0), int(p["duplicate_h"] > 0), int(p["duplicate_c"] > 0)]
        self.tail = p["n_sin_waves"] + sum(self.goals)
        self.widths = [[pp + self.tail] + list(r.hidden) + [o] for r, pp, o in zip(robots, self.pos_pad, self.nout)]
        self.wmax = [max(w[l] for w in self.widths) for l in range(len(self.widths[0]))]
        base = np.arange(self.R) * self.wmax[0]
        self.in_pos = _idx(np.concatenate([b + np.arange(3 * n) for b, n in zip(base, nv)]))
        self.in_tail = _idx(np.concatenate([b + pp + np.arange(self.tail) for b, pp in zip(base, self.pos_pad)]))
        self.out_rows = _idx(np.concatenate([r * self.wmax[-1] + np.arange(o) for r, o in enumerate(self.nout)]))
        self.drag = math.exp(-p["dt"] * p["drag_damping"])
        self.fn = {"tanh": torch.tanh, "sin": torch.sin}

    def per_robot(self, a):
        if self.R == 1:
            return a.sum(0, keepdim=True)
        return torch.zeros((self.R,) + a.shape[1:], dtype=a.dtype, device=a.device).index_add(0, self.rob, a)

    def center(self, x):
        return self.per_robot(x) / self.n

    def compact(self, r, full):
        """First-layer weights in the compact column order: positions, sines, one column per goal value."""
        p, N = self.p, self.robots[r].n_vertices
        s = p["n_sin_waves"]
        q = s + 6 * N
        parts = [full[:, s:q].reshape(-1, N, 2, 3)[:, :, 0].reshape(-1, 3 * N)]
        parts.append(full.new_zeros(full.shape[0], self.pos_pad[r] - 3 * N))
        parts.append(full[:, :s])
        if p["duplicate_v"]:
            parts.append(full[:, q:q + 2 * p["duplicate_v"]].reshape(-1, p["duplicate_v"], 2).sum(1))
        q += 2 * p["duplicate_v"]
        for key in ("duplicate_h", "duplicate_c"):
            if p[key]:
                parts.append(full[:, q:q + p[key]].sum(1, keepdim=True))
            q += p[key]
        return torch.cat(parts, 1)

    def full_cols(self, r):
        p = self.p
        return p["n_sin_waves"] + 6 * self.robots[r].n_vertices + 2 * p["duplicate_v"] + p["duplicate_h"] + p["duplicate_c"]

    def set_weights(self, weights):
        """weights[r][l] = (W in the reference layout, b or None)."""
        self.W, self.b = [], []
        for l in range(len(self.wmax) - 1):
            W = torch.zeros(self.R, self.wmax[l + 1], self.wmax[l], dtype=torch.float64, device="cuda")
            b = torch.zeros(self.R, self.wmax[l + 1], 1, dtype=torch.float64, device="cuda")
            for r in range(self.R):
                w, bias = weights(r, l)
                w = self.compact(r, w) if l == 0 else w
                W[r, :w.shape[0], :w.shape[1]] = w
                if bias is not None:
                    b[r, :bias.shape[0], 0] = bias
            self.W.append(W)
            self.b.append(b)

    def init_weights(self, seed):
        L = len(self.wmax) - 1

        def one(r, l):
            rows, cols = self.widths[r][l + 1], self.full_cols(r) if l == 0 else self.widths[r][l]
            return (_uniform(seed, r * L + l, rows * cols).view(rows, cols) * 2 - 1) * math.sqrt(6.0 / cols), None
        self.set_weights(one)

    def goal_rows(self, t, tv, th, tc):
        """[R * tail, E] sine and goal inputs of substep t."""
        p = self.p
        s = _t64(np.sin(p["spring_omega"] * t * p["dt"] + 2 * np.pi / max(1, p["n_sin_waves"]) * np.arange(p["n_sin_waves"])))
        rows = [s[None, :, None].expand(self.R, -1, self.E)]
        if self.goals[0]:
            rows.append(torch.stack([tv[t, :, :, 0], tv[t, :, :, 2]], 1) / p["max_speed"])
        if self.goals[1]:
            rows.append(th[t][:, None])
        if self.goals[2]:
            rows.append(tc[t][:, None])
        return torch.cat(rows, 1).reshape(-1, self.E)

    def inputs(self, x, c, tail):
        xin = torch.zeros(self.R * self.wmax[0], self.E, dtype=torch.float64, device="cuda")
        pos = ((x - c[self.rob]) / ACT_SCALE).permute(0, 2, 1).reshape(-1, self.E)
        return xin.index_copy(0, self.in_pos, pos).index_copy(0, self.in_tail, tail)

    def controller(self, x, c, tail, *wb):
        a = self.inputs(x, c, tail).view(self.R, self.wmax[0], self.E)
        L = len(wb) // 2
        for l in range(L):
            act = self.fn[self.p["activation_output" if l == L - 1 else "activation_hidden"]]
            a = act(torch.baddbmm(wb[L + l].expand(-1, -1, self.E), wb[l], a))
        return a.reshape(-1, self.E)[self.out_rows]

    def advance(self, x, v, out):
        """One substep with controller outputs `out` [O, E]."""
        p, dt = self.p, self.p["dt"]
        act = torch.cat([out, out.new_zeros(1, out.shape[1])])[self.out]
        return self.substep(x, v, act)

    def substep(self, x, v, act):
        p, dt = self.p, self.p["dt"]
        d, dv = x[self.sa] - x[self.sb], v[self.sa] - v[self.sb]
        n2 = (d * d).sum(-1)
        length = torch.sqrt(n2 + 1e-8) + 1e-4
        target = self.len * (1 + self.coef * act)
        nrm = d / torch.sqrt(n2)[..., None]
        vrel = (dv * nrm).sum(-1)
        imp = (dt * (length - target) * self.k / length)[..., None] * d + (p["dashpot_damping"] * vrel)[..., None] * nrm
        vinc = torch.zeros_like(v).index_add(0, self.sa, -imp).index_add(0, self.sb, imp)
        g = torch.tensor([0.0, dt * p["gravity"], 0.0], dtype=torch.float64, device="cuda")
        ov = self.drag * v + g + vinc
        hit = (x[..., 1] + dt * ov[..., 1] < p["ground_height"]) & (ov[..., 1] < -1e-4)
        vy = torch.where(hit, ov[..., 1], torch.full_like(ov[..., 1], -1.0))
        toi = torch.where(hit, -(x[..., 1] - p["ground_height"]) / vy, torch.zeros_like(vy))
        f = p["friction"] * -vy

        def slide(u):
            s = torch.where(u < 0, torch.clamp(u + f, max=0.0), torch.clamp(u - f, min=0.0))
            return torch.where(hit, s, u)
        nv = torch.stack([slide(ov[..., 0]), torch.where(hit, torch.zeros_like(vy), ov[..., 1]), slide(ov[..., 2])], -1)
        return x + toi[..., None] * ov + (dt - toi)[..., None] * nv, nv

    def rollout(self, x, v, steps, tv, th, tc, grad):
        """x, v after every substep t < steps and the outputs of each: xs[0..steps], outs[0..steps-1]."""
        wb = self.W + self.b
        xs, outs = [x], []
        for t in range(steps):
            tail = self.goal_rows(t, tv, th, tc)

            def one(x, v, tail, *wb):
                out = self.controller(x, self.center(x), tail, *wb)
                return self.advance(x, v, out) + (out,)
            x, v, out = checkpoint(one, x, v, tail, *wb, use_reentrant=False) if grad else one(x, v, tail, *wb)
            xs.append(x)
            outs.append(out)
        return xs, v, outs

    def heights(self, xs):
        """Running height and upper height [t][E] (one robot type)."""
        hs, us, h = [], [], None
        for t, x in enumerate(xs):
            lo = x[..., 1].min(0).values
            h = lo if t % self.p["jump_period"] == 0 else torch.maximum(h, lo)
            hs.append(h)
            us.append(x[..., 1].max(0).values)
        return hs, us

    def losses(self, xs, outs, steps, T, tv, th, tc, mask):
        """[8][R, E]: total and the terms in the library's order; the rollout
        ran substeps 0 .. steps - 2, so xs holds x[0 .. steps - 1]; what was
        never computed reads as zero."""
        p, B = self.p, self.E
        zero = torch.zeros(self.R, self.E, dtype=torch.float64, device="cuda")
        rp, tp, jp = p["run_period"], p["turn_period"], p["jump_period"]
        cs = [self.center(x) for x in xs[:steps - 1]]
        c0 = torch.zeros(self.R, self.E, 3, dtype=torch.float64, device="cuda")
        x_at = lambda t: xs[t] if t < steps else torch.zeros_like(xs[0])  # noqa: E731
        c_at = lambda t: cs[t] if t < steps - 1 else c0  # noqa: E731
        terms = {k: zero for k in ("velocity", "height", "pose", "rotation", "weight", "actuation", "crawl")}
        if "height" in mask:
            hs, us = self.heights(xs[:steps - 1])
        o_h = lambda s, t: s[t][None] if t < steps - 1 else zero  # noqa: E731
        for t in range(min(steps, T - 1) + 1):
            if t % tp > rp:
                u = t - rp
                e = c_at(t) - c_at(u) - tv[u]        # the velocity and rotation terms share their window
                terms["velocity"] = terms["velocity"] + (e[..., 0] ** 2 + e[..., 2] ** 2) / B / steps * 100
                ang = th[u] * 72.0 / 180.0 * 3.1415926535
                ca, sn = torch.cos(ang)[self.rob], torch.sin(ang)[self.rob]
                a, b = x_at(t) - c_at(t)[self.rob], x_at(u) - c_at(u)[self.rob]
                ex = a[..., 0] - (ca * b[..., 0] - sn * b[..., 2])
                ey, ez = a[..., 1] - b[..., 1], a[..., 2] - (sn * b[..., 0] + ca * b[..., 2])
                terms["rotation"] = terms["rotation"] + self.per_robot(ex * ex + ey * ey + ez * ez) / steps / 40
            if "height" not in mask:
                continue
            if t >= 1 and t % jp == jp - 1:
                d = o_h(hs, t) - th[t]
                terms["height"] = terms["height"] + torch.where(th[t] > 0.1 + 1e-6, d * d, zero) / B / (steps // jp) * 100
            if t >= 1:
                d = torch.clamp(o_h(us, t) - 0.1, min=0.0)
                terms["crawl"] = terms["crawl"] + torch.where(tc[t] > 1 - 1e-4, d * d, zero) / B / steps * 5
            if t >= 1 and t % jp == 0:
                terms["pose"] = terms["pose"] + ((x_at(t) - xs[0].detach()) ** 2).sum((0, 2))[None] / B / (steps // jp)
            if t < steps - 1:
                lim = torch.sqrt(tv[t, :, :, 0].abs() / 0.08)
                a = torch.cat([outs[t], outs[t].new_zeros(1, self.E)])[self.out].abs()
                s = torch.clamp(a - lim, min=0.0).sum(0, keepdim=True)
                terms["actuation"] = terms["actuation"] + torch.where(th[t] < 0.1 + 1e-4, s, zero) / self.ns[0] / B / steps * 10
        rows = [terms[k] if k in mask else zero
                for k in ("velocity", "height", "pose", "rotation", "weight", "actuation", "crawl")]
        return torch.stack([sum(rows)] + rows)

    def train(self, x0, v0, steps, T, tv, th, tc, mask):
        """losses [8][R, E] and the gradients of every layer's padded W and b."""
        for a in self.W + self.b:
            a.requires_grad_(True)
        xs, _, outs = self.rollout(x0, v0, steps - 1, tv, th, tc, True)
        loss = self.losses(xs, outs, steps, T, tv, th, tc, mask)
        loss[0].sum().backward()
        return loss.detach(), xs[-1].detach(), [w.grad for w in self.W], [b.grad for b in self.b]

    def packed(self, gW, gb):
        """The library's gradient buffers: robot after robot, layer after layer,
        rows padded to 4 values, each weight block to 8, each bias block to 4."""
        ws, bs = [], []
        size = lambda n, m: -(-n // m) * m  # noqa: E731
        w_total = b_total = 0
        for w in self.widths:
            for l in range(len(w) - 1):
                w_total += size(w[l + 1] * size(w[l], 4), 8)
                b_total += size(w[l + 1], 4)
        ws, bs = (torch.zeros(n, dtype=torch.float64, device="cuda") for n in (w_total, b_total))
        w0 = b0 = 0
        for r, w in enumerate(self.widths):
            for l in range(len(w) - 1):
                pitch = size(w[l], 4)
                ws[w0:w0 + w[l + 1] * pitch].view(w[l + 1], pitch)[:, :w[l]] = gW[l][r, :w[l + 1], :w[l]]
                bs[b0:b0 + w[l + 1]] = gb[l][r, :w[l + 1], 0]
                w0 += size(w[l + 1] * pitch, 8)
                b0 += size(w[l + 1], 4)
        return [ws, bs]

    def field(self, a):
        """Env-after-env rows [envs x vertices][3] to [V, E, 3]."""
        parts, at = [], 0
        for r in self.robots:
            n = r.n_vertices * self.E
            parts.append(_t64(a[at:at + n]).view(self.E, r.n_vertices, 3).transpose(0, 1))
            at += n
        return torch.cat(parts)

    def rows(self, f):
        parts, at = [], 0
        for r in self.robots:
            parts.append(f[at:at + r.n_vertices].transpose(0, 1).reshape(-1, 3))
            at += r.n_vertices
        return torch.cat(parts)


def exact(case, seed):
    out = globals()["_exact_" + case["kind"]](dict(case), int(seed))
    torch.cuda.empty_cache()
    return out


def _model(case, T, seed):
    robots, envs = _robots(case)
    m = _Model(robots, envs, _params(case, T, T))
    m.init_weights(seed + 2)
    tg = [_t64(a).view((T, m.R, m.E) + a.shape[2:]) for a in _targets(case, T, m.R * m.E, seed)]
    x0, v0 = (m.field(a) for a in _state(robots, envs, seed, _lift(case), case["kind"] == "eval"))
    return m, x0, v0, tg


def _exact_train(case, seed):
    T = case["steps"]
    m, x0, v0, tg = _model(case, T, seed)
    loss, _, gW, gb = m.train(x0, v0, T, T, *tg, m.p["loss"])
    return dict(loss=(loss * m.E).reshape(8, -1).cpu().numpy(), grads=m.packed(gW, gb))


def _observed(m, xs):
    """center [t][E][3], running height, upper height, rotation [t][E] (one robot type)."""
    c = torch.stack([m.center(x)[0] for x in xs])
    h, u = (torch.stack(s) for s in m.heights(xs))
    head = (xs[0][..., 0] < c[0][None, :, 0]).double()
    rot = []
    for x in xs:
        nh, nt = head.sum(0), (1 - head).sum(0)
        d = ((1 - head)[..., None] * x).sum(0) * nh[:, None] - (head[..., None] * x).sum(0) * nt[:, None]
        rot.append(torch.atan2(d[:, 2], d[:, 0]))
    return dict(center=c, height=h, upper_height=u, rotation=torch.stack(rot))


def _exact_eval(case, seed):
    T = case["steps"] + 2
    m, x0, v0, tg = _model(case, T, seed)
    with torch.no_grad():
        xs, v, _ = m.rollout(x0, v0, case["steps"] + 1, *tg, False)
        obs = _observed(m, xs[:-1])
    out = {k: torch.cat([a, torch.zeros_like(a[:1])]).cpu().numpy() for k, a in obs.items()}
    out["x"], out["v"] = m.rows(xs[-1]).cpu().numpy(), m.rows(v).cpu().numpy()
    return out


def _exact_gym(case, seed):
    robot, E, n = _robot(case["robot"]), case["envs"], case["steps"]
    m = _Model([robot], E, _params(case, n + 2, n))
    x = _t64(_state([robot], 1, seed)[0])[:, None].expand(-1, E, -1).contiguous()
    v = torch.zeros_like(x)
    tv, th, tc = (torch.zeros((n + 2, 1, E) + s, dtype=torch.float64, device="cuda") for s in ((3,), (), ()))
    th[:] = 0.1            # the goal that reset() sets
    acts = _t64(_actions(case, seed))
    springs = _idx(np.nonzero(robot.springs[:, 4] > 0)[0])
    xs = [x]
    for t in range(n):
        out = torch.zeros(m.O, E, dtype=torch.float64, device="cuda")
        out[m.out[springs]] = acts[t].T
        x, v = m.advance(x, v, out)
        xs.append(x)
    obs, s = [], m.p["n_sin_waves"]
    for t, x in enumerate(xs):
        rel = (x - m.center(x)[m.rob]) / ACT_SCALE
        body = torch.cat([rel, torch.zeros_like(rel)], -1).permute(1, 0, 2).reshape(E, -1)
        tail = m.goal_rows(t, tv, th, tc).T
        obs.append(torch.cat([tail[:, :s], body, tail[:, s:]], 1).reshape(-1).clamp(-1, 1))
    seen = _observed(m, xs)
    c, h = seen["center"][..., 0].cpu().numpy(), seen["height"].cpu().numpy()
    rewards, last = [], np.full(E, 0.1)
    for t in range(1, n + 1):
        rv = np.zeros(E)
        for i in range(t):
            tar = c[i]
            rv += ((c[t - 1] - tar) ** 2 - (c[t] - tar) ** 2) / m.p["max_speed"] ** 2 / 400.0
        rh = -((h[t] - 0.1) ** 2 - (last - 0.1) ** 2) / 0.1 ** 2 * 10.0
        last = np.maximum(last, h[t])
        rewards.append((rv + rh).sum() / E)
    return dict(obs=torch.stack(obs).cpu().numpy(), reward=np.array(rewards))


def _exact_serve(case, seed):
    T, W = case["max_steps"], _serve_weights(case, seed)
    losses, final, grads = [], [], []
    for r in _serve_requests(case, seed):
        robot = _serve_robots(case)[r["kind"]]
        m = _Model([robot], 1, _params(case, T, T))
        m.set_weights(lambda _, l: tuple(_t64(a) for a in W[r["kind"]][l]))
        tg = [_t64(a)[:, None, None] for a in (r["tv"], r["th"], np.zeros(T))]
        x0 = m.field(r["x0"])
        if r["grad"]:
            loss, x, gW, gb = m.train(x0, torch.zeros_like(x0), r["steps"], T, *tg, m.p["loss"])
            g0 = torch.zeros(robot.hidden[0], m.full_cols(0), dtype=torch.float64, device="cuda")
            s, N = m.p["n_sin_waves"], robot.n_vertices
            pos = g0[:, s:s + 6 * N].view(-1, N, 2, 3)
            pos[:, :, 0] = gW[0][0, :, :3 * N].reshape(-1, N, 3)
            tail = gW[0][0, :, m.pos_pad[0]:]
            g0[:, :s], g0[:, s + 6 * N:] = tail[:, :s], tail[:, s:]
            for l in range(len(gW)):
                grads += [(g0 if l == 0 else gW[l][0]).reshape(-1), gb[l][0].reshape(-1)]
        else:
            with torch.no_grad():
                xs, _, outs = m.rollout(x0, torch.zeros_like(x0), r["steps"] - 1, *tg, False)
                loss, x = m.losses(xs, outs, r["steps"], T, *tg, m.p["loss"]), xs[-1]
        losses.append(loss.reshape(8))
        final.append(x.reshape(-1))
    return dict(loss=torch.stack(losses).cpu().numpy(), x=torch.cat(final).cpu().numpy(), grad=torch.cat(grads).cpu().numpy())


def _exact_advance(case, seed):
    robot, x0, v0, act = _advance_inputs(case, seed)
    m = _Model([robot], case["envs"], _params(case, 2, 2))
    x, v = _t64(x0).transpose(0, 1).contiguous(), _t64(v0).transpose(0, 1).contiguous()
    a = _t64(act).T.contiguous()
    for _ in range(case["steps"]):
        x, v = m.substep(x, v, a)
    return dict(x=x.transpose(0, 1).contiguous(), v=v.transpose(0, 1).contiguous())


def _exact_mpm(case, seed):
    pos, mus, fib, M, p = _mpm_body(case)
    x0, v0, act, w, target = _mpm_inputs(case, seed)
    D, E, n, T = case["dim"], case["envs"], p["n_grid"], case["steps"]
    dx, dt, P = 1.0 / n, p["dt"], pos.shape[0]
    fib = np.tile(np.eye(D)[1], (P, 1)) if fib is None else fib
    eye = torch.eye(D, dtype=torch.float64, device="cuda")
    f, active = _t64(fib), _t64((mus >= 0).astype(float))
    muscle = _idx(np.maximum(mus, 0))
    offs = torch.stack(torch.meshgrid(*[torch.arange(3, device="cuda")] * D, indexing="ij"), -1).view(-1, D)
    stride = _idx([n ** (D - 1 - d) for d in range(D)])
    cell = torch.stack(torch.meshgrid(*[torch.arange(n, device="cuda")] * D, indexing="ij"), -1).view(-1, D)
    inside = (~((cell < p["bound"]) | (cell > n - p["bound"])).any(1)).double()[:, None]
    env = torch.arange(E, device="cuda")[:, None] * n ** D
    g = torch.zeros(D, dtype=torch.float64, device="cuda")
    g[1] = dt * p["gravity"]
    ks = dt * p["p_vol"] * 4 / dx / dx

    def step(x, v, C, F, a):
        base = (x.detach() / dx - 0.5).floor()
        fx = x / dx - base
        wt = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2])
        nF = (eye + dt * C) @ F
        J = torch.linalg.det(nF)
        if p["material"] == "fixed_corotated":
            c, s = nF[..., 0, 0] + nF[..., 1, 1], nF[..., 1, 0] - nF[..., 0, 1]
            r = torch.sqrt(c * c + s * s)
            c, s = c / r, s / r
            R = torch.stack([torch.stack([c, -s], -1), torch.stack([s, c], -1)], -2)
            tau = 2 * p["mu"] * (nF - R) @ nF.mT + (p["la"] * (J - 1) * J)[..., None, None] * eye
        else:
            tau = p["mu"] * (nF @ nF.mT - eye) + (p["la"] * torch.log(J))[..., None, None] * eye
        u = (nF @ f[..., None])[..., 0]
        tau = tau + (a[:, muscle] * active * p["act_strength"])[..., None, None] * u[..., :, None] * u[..., None, :]
        aff = -ks * tau + p["mass"] * C
        gm = torch.zeros(E * n ** D, D + 1, dtype=torch.float64, device="cuda")
        idx, wts, dps = [], [], []
        for o in offs:
            wq = 1.0
            for d in range(D):
                wq = wq * wt[o[d], ..., d]
            dp = o.double() - fx
            i = ((base.long() + o) * stride).sum(-1) + env
            mom = p["mass"] * v + (aff @ (dp * dx)[..., None])[..., 0]
            val = torch.cat([wq[..., None] * mom, wq[..., None] * p["mass"]], -1)
            gm = gm.index_add(0, i.reshape(-1), val.reshape(-1, D + 1))
            idx.append(i)
            wts.append(wq)
            dps.append(dp)
        gv = (gm[:, :D] / (gm[:, D:] + 1e-10) + g) * inside.repeat(E, 1)
        nv, nC = torch.zeros_like(v), torch.zeros_like(C)
        for i, wq, dp in zip(idx, wts, dps):
            gq = wq[..., None] * gv[i]
            nv = nv + gq
            nC = nC + 4 / dx * gq[..., :, None] * dp[..., None, :]
        return x + dt * nv, nv, nC, nF

    x, v = _t64(x0), _t64(v0)
    C = torch.zeros(E, P, D, D, dtype=torch.float64, device="cuda")
    F = eye.expand(E, P, D, D).contiguous()
    a = _t64(act).requires_grad_(case["grad"])
    centers = [x.mean(1)]
    for t in range(T):
        x, v, C, F = checkpoint(step, x, v, C, F, a[t], use_reentrant=False) if case["grad"] else step(x, v, C, F, a[t])
        centers.append(x.mean(1))
    centers = torch.stack(centers)
    loss = (_t64(w)[:, None, None] * (centers - _t64(target)) ** 2).sum()
    out = dict(loss=loss.detach().cpu().numpy(), centers=centers.detach().cpu().numpy())
    if not case["grad"]:
        return dict(out, x=x.cpu().numpy(), v=v.cpu().numpy())
    loss.backward()
    return dict(out, act=a.grad.cpu().numpy())
