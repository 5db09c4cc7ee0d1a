"""Clusters per environment against one CTA per environment.

A small batch runs its fused kernels with one thread-block cluster per env;
``simulate(per_env=True)`` runs the same rollout with the single-CTA kernels,
one launch per env, here with the springs evaluated at both endpoints as the
clusters do (a per-spring table contracts an FP64 impulse's products the other
way round, one ulp apart).  The forward pass sums every row, vertex and centre in
the same order in both, so observables and final state are the same bits; the
reverse pass sums the controller's transposed products in another order, so
gradients agree within the configuration's bar (FP64 rel 1e-8, FP32 rel 1e-4).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(n, hidden, seed=0, outputs=True):
    from cls_b200 import robot_design
    from cls_b200.batch import Robot
    o, s = robot_design.random_lattice(np.random.default_rng(seed), n)
    return Robot.actuated_outputs(o, s, hidden=list(hidden)) if outputs else Robot(o, s, hidden=list(hidden))


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


CASES = [
    # (vertices, hidden widths, envs of each robot, steps, K, one output per actuated spring)
    ((8,), (4,), 1, 7, 7, True),              # one cube: fewer vertices than CTAs x lanes
    ((60,), (64,), 1, 61, 20, True),          # several segments, replayed recompute
    ((60, 250, 700), (128, 128), 1, 41, 50, True),
    ((93,), (37, 21, 5), 3, 23, 9, False),    # odd widths, three hidden layers, an output per spring
    ((2000,), (128, 128), 1, 9, 4, True),     # largest robot: incidence records and both state copies fill the CTA
    ((120,), (64,), 40, 21, 50, True),        # clusters of 2 or 4
    ((40,), (600,), 2, 12, 5, True),          # a hidden layer wider than the block
]


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_cluster_equals_single_cta(case, precision):
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch
    sizes, hidden, envs, steps, K, outputs = CASES[case]
    if precision == 64 and max(sizes) > 1000:
        pytest.skip("a 2000-vertex robot in FP64 exceeds one CTA's shared memory")
    robots = [_lattice(n, hidden, seed=n, outputs=outputs) for n in sizes]
    loss = ("velocity", "rotation", "height", "pose", "actuation", "crawl")
    p = cls_b200.default_params(**workloads._params(steps, K, precision=precision, run_period=5, turn_period=30,
                                                    jump_period=4, loss=loss))
    b = MassSpringBatch(robots, [r for r in range(len(robots)) for _ in range(envs)], p)
    rng = np.random.default_rng(case)
    try:
        b.weights_init(3)
        b.set_spring_tables(0)
        E, T = b.n_envs, b.T
        tv, th = workloads.targets(rng, T, E)
        tc = np.zeros((T, E))
        tc[:, ::2] = 1.0
        b.set_targets(tv, th + 0.15, tc)
        x0 = np.concatenate([np.tile(r.objects, (envs, 1)) for r in robots])
        x0[:, 1] -= 0.09                       # the first contacts come within a few substeps
        b.set_state(x0 + rng.uniform(-2e-3, 2e-3, x0.shape), rng.uniform(-0.1, 0.1, x0.shape))

        def one(per_env):
            b.simulate(steps, per_env=per_env)
            terms, env = b.loss()
            grads = [a for r in range(len(robots)) for l in range(b.n_layers(r)) for a in b.get_grads(r, l)]
            return b.observables(), b.final_state(), env, grads, b.state_grads()
        ref, got = one(True), one(False)
    finally:
        b.close()
    for k in ("center", "height", "upper_height"):
        assert np.array_equal(got[0][k], ref[0][k]), k
    assert np.abs(got[0]["rotation"] - ref[0]["rotation"]).max() <= (1e-4 if precision == 32 else 1e-9)
    for g, r in zip(got[1], ref[1]):
        assert np.array_equal(g, r)
    assert np.array_equal(got[2], ref[2])
    tol = 1e-8 if precision == 64 else 1e-4
    for g, r in zip(got[3] + list(got[4]), ref[3] + list(ref[4])):
        assert np.isfinite(g).all()
        assert _rel(g, r) < tol


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("graph", [False, True])
def test_heaviest_on_clusters_beside_single_ctas(graph, precision):
    """Few heavy envs among many light ones: the heavy ones run as clusters in a
    launch beside that of the others.  Same bars as above; a captured step replays
    the same two launches."""
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch
    import torch
    steps, K = 15, 6
    robots = [_lattice(n, (32, 16), seed=n) for n in (700, 30)]
    p = cls_b200.default_params(**workloads._params(steps, K, precision=precision, run_period=5, turn_period=30,
                                                    jump_period=4, loss=("velocity", "rotation", "height")))
    b = MassSpringBatch(robots, [0] * 4 + [1] * 196, p)
    rng = np.random.default_rng(5)
    try:
        b.set_controller_path("per_env")
        b.weights_init(3)
        b.set_spring_tables(0)
        tv, th = workloads.targets(rng, b.T, b.n_envs)
        b.set_targets(tv, th + 0.15, np.zeros((b.T, b.n_envs)))
        x0 = np.concatenate([robots[0].objects] * 4 + [robots[1].objects] * 196)
        x0[:, 1] -= 0.09
        b.set_state(x0 + rng.uniform(-2e-3, 2e-3, x0.shape), rng.uniform(-0.1, 0.1, x0.shape))

        def read():
            return b.final_state(), [a for r in (0, 1) for l in range(b.n_layers(r)) for a in b.get_grads(r, l)]

        def run(per_env):
            b.simulate(steps, per_env=per_env)
            b.loss()
            return read()
        ref = run(True)
        if graph:
            s = torch.cuda.Stream()
            b.set_stream(s.cuda_stream)
            b.graph_capture(steps, False)
            for _ in range(2):
                b.graph_launch(0)
            torch.cuda.synchronize()
            got = read()
        else:
            got = run(False)
    finally:
        b.close()
    for g, r in zip(got[0], ref[0]):
        assert np.array_equal(g, r)
    tol = 1e-8 if precision == 64 else 1e-4
    for g, r in zip(got[1], ref[1]):
        assert np.isfinite(g).all()
        assert _rel(g, r) < tol
