"""Spring tables of robots with hub vertices (more springs than a thread's list holds):
the bits of the direct gathers, on by default, and never slower than those."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _robot(n_v, hubs, rest, seed=1, parallel=1):
    """hubs[i] springs from vertex i to later vertices, `rest` springs among the others;
    `parallel` copies of every spring."""
    from cls_b200.batch import Robot
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.05, 0.6, (n_v, 3))
    pairs = []
    for h, deg in enumerate(hubs):
        pairs += [(h, j) if j % 2 else (j, h) for j in len(hubs) + np.arange(deg) % (n_v - len(hubs))]
    while len(pairs) < sum(hubs) + rest:
        i, j = rng.integers(len(hubs), n_v, 2)
        if i != j:
            pairs.append((int(i), int(j)))
    pairs = [p for p in pairs for _ in range(parallel)]
    pairs = [pairs[k] for k in rng.permutation(len(pairs))]
    s = np.array([[i, j, np.linalg.norm(x[i] - x[j]), 3e3, 0.2 if k % 3 else 0.0] for k, (i, j) in enumerate(pairs)])
    return Robot.actuated_outputs(x, s, hidden=[16])


def _batch(robots, envs, precision, steps=13, path="per_env"):
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch
    b = MassSpringBatch(robots, envs, cls_b200.default_params(
        **workloads._params(steps, 5, precision=precision, run_period=3, turn_period=20)))
    b.set_controller_path(path)
    b.weights_init(1)
    b.set_targets(*workloads.targets(np.random.default_rng(2), b.T, b.n_envs))
    return b


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("threads", [64, 256, 512, 1024])
@pytest.mark.parametrize("n_v, hubs, rest, parallel", [
    (60, (48,), 60, 1),                        # the longest list of one thread
    (60, (49, 48, 50), 60, 1),
    (120, (64, 65, 80, 81, 96, 113), 100, 1),  # around whole leaves; more hubs than half-warps of a CTA of 64
    (2, (), 1, 60),                            # nothing but hubs
    (6, (), 15, 24),                           # every vertex a hub
    (300, (299,), 0, 1),                       # a star
])
def test_tables_equal_direct_gathers(n_v, hubs, rest, parallel, threads, precision):
    robots = [_robot(n_v, hubs, rest, parallel=parallel), _robot(20, (), 40)]
    out = []
    for mode in (0, 1):
        b = _batch(robots, [0, 1, 0], precision)
        try:
            b.set_spring_tables(mode)
            b.set_launch_shape(threads, 1)
            b.simulate(13, per_env=True)
            out.append([b.observables()["center"], *b.final_state(), *b.state_grads(),
                        *(a for r in range(2) for l in range(2) for a in b.get_grads(r, l))])
        finally:
            b.close()
    for u, w in zip(*out):
        assert np.isfinite(u).all() and np.array_equal(u, w)


def test_batched_controller():
    robot = _robot(120, (92, 60), 300)
    out = []
    for mode in (0, 1):
        b = _batch([robot], [0] * 40, 32, path="batched")
        try:
            b.set_spring_tables(mode)
            b.simulate(13)
            out.append([*b.final_state(), *b.state_grads()])
        finally:
            b.close()
    for u, w in zip(*out):
        assert np.isfinite(u).all() and np.array_equal(u, w)


@pytest.mark.parametrize("path", ["per_env", "batched"])
@pytest.mark.parametrize("degree", [60, 200])
def test_on_by_default_and_not_slower(degree, path):
    """A batch of 600 robots with a hub: tables by default, and within 5 % of the direct
    gathers or faster (0.7 to 0.8 of their time before a rule on degrees kept such
    batches off the tables)."""
    import torch
    b = _batch([_robot(max(120, degree + 1), (degree,), 420)], [0] * 600, 32, 42, path)
    try:
        assert b.spring_tables
        b.set_stream(torch.cuda.current_stream().cuda_stream)
        times = {}
        for mode in (-1, 0):
            b.set_spring_tables(mode)
            t = []
            for _ in range(9):
                ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                ev[0].record()
                b.simulate(41)
                ev[1].record()
                torch.cuda.synchronize()
                t.append(ev[0].elapsed_time(ev[1]))
            times[mode] = np.median(t[2:])
        assert times[-1] < 1.05 * times[0]
    finally:
        b.close()


def test_one_robot_keeps_its_tables():
    """One robot: on a cluster, which evaluates a vertex's springs by a half-warp, only
    while no vertex has very many (a hub of 92 springs 1.06 of the single CTA's time, of
    400 1.22)."""
    for degree, clusters in ((24, True), (92, False), (200, False)):
        b = _batch([_robot(max(120, degree + 1), (degree,), 420)], [0], 32)
        assert (b.clusters[0] > 1) == clusters
        b.set_spring_tables(0)
        assert b.clusters[0] > 1         # both forms evaluate the hub's springs by a half-warp
        b.close()


def test_policy_steps():
    """Steps with outputs from outside: the same observations with tables and without."""
    from cls_b200._capi import ptr
    out = []
    for mode in (-1, 0):
        b = _batch([_robot(120, (92, 60), 300), _robot(20, (), 40)], [0, 1], 32)
        try:
            b.set_spring_tables(mode)
            rng = np.random.default_rng(3)
            obs, aux, act = np.zeros(4096), np.zeros(8), rng.uniform(-1, 1, 4096)
            seen = []
            for t in range(6):
                b._c(b.lib.cls_env_step(b.h, t, ptr(act) if t else None, ptr(obs), ptr(aux)))
                seen += [obs.copy(), aux.copy()]
            out.append(seen)
        finally:
            b.close()
    assert not np.array_equal(out[0][0], out[0][-2])
    for u, w in zip(*out):
        assert np.isfinite(u).all() and np.array_equal(u, w)
