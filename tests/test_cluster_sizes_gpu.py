"""Every cluster size (cls_set_clusters) against one CTA per env, on the cases of
test_cluster_gpu and with its bars: the forward pass computes the same bits, whether
the single CTA takes its springs from a table or from both endpoints; gradients agree
within FP64 rel 1e-8, FP32 rel 1e-4."""
import numpy as np
import pytest

from test_cluster_gpu import CASES, _lattice, _rel

pytestmark = pytest.mark.gpu


def _batch(sizes, hidden, envs, steps, K, outputs, precision, seed=0):
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch
    robots = [_lattice(n, hidden, seed=n, outputs=outputs) for n in sizes]
    loss = ("velocity", "rotation", "height", "pose", "actuation", "crawl")
    b = MassSpringBatch(robots, [r for r, n in enumerate(envs) for _ in range(n)], cls_b200.default_params(
        **workloads._params(steps, K, precision=precision, run_period=5, turn_period=30, jump_period=4, loss=loss)))
    b.set_controller_path("per_env")
    rng = np.random.default_rng(seed)
    b.weights_init(3)
    tv, th = workloads.targets(rng, b.T, b.n_envs)
    tc = np.zeros((b.T, b.n_envs))
    tc[:, ::2] = 1.0
    b.set_targets(tv, th + 0.15, tc)
    x0 = np.concatenate([np.tile(r.objects, (n, 1)) for r, n in zip(robots, envs)])
    x0[:, 1] -= 0.09                       # the first contacts come within a few substeps
    b.set_state(x0 + rng.uniform(-2e-3, 2e-3, x0.shape), rng.uniform(-0.1, 0.1, x0.shape))
    return b


def _run(b, steps, per_env):
    b.simulate(steps, per_env=per_env)
    _, env = b.loss()
    o = b.observables()
    same = [o["center"], o["height"], o["upper_height"], *b.final_state(), env]
    grads = [a for r in range(len(b.robots)) for l in range(b.n_layers(r)) for a in b.get_grads(r, l)]
    return same, grads + list(b.state_grads())


def _compare(got, ref, precision):
    for g, r in zip(got[0], ref[0]):
        assert np.array_equal(g, r)
    tol = 1e-8 if precision == 64 else 1e-4
    for g, r in zip(got[1], ref[1]):
        assert np.isfinite(g).all()
        assert _rel(g, r) < tol


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_every_size(case, precision):
    sizes, hidden, envs, steps, K, outputs = CASES[case]
    if precision == 64 and max(sizes) > 1000:
        pytest.skip("a 2000-vertex robot in FP64 exceeds one CTA's shared memory")
    from cls_b200 import _capi
    b = _batch(sizes, hidden, [envs] * len(sizes), steps, K, outputs, precision, case)
    try:
        ran = []
        for tables in (-1, 0):
            b.set_spring_tables(tables)
            ref = _run(b, steps, True)
            for size in (1, 2, 4, 8, 16):
                b.set_clusters(-1)
                before = b.clusters
                try:
                    b.set_clusters(size)
                except _capi.ClsError:
                    assert b.clusters == before and max(sizes) > 500    # a large robot's share of two or four
                    continue
                assert b.clusters == ((size, b.n_envs) if size > 1 else (1, 0))
                _compare(_run(b, steps, False), ref, precision)
                ran.append(size)
        assert {8, 16} <= set(ran)
    finally:
        b.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("size, heavy", [(2, 1), (4, 4), (8, 3), (16, 4), (4, 60)])
def test_heaviest_beside_the_others(size, heavy, precision):
    """`heavy` envs on clusters beside the rest on single CTAs; a captured step keeps
    its clusters."""
    import torch
    steps = 15
    b = _batch((300, 30), (32, 16), (4, 66), steps, 6, True, precision)
    try:
        ref = _run(b, steps, True)
        b.set_clusters(size, heavy)
        assert b.clusters == (size, heavy)
        _compare(_run(b, steps, False), ref, precision)
        b.set_stream(torch.cuda.Stream().cuda_stream)
        b.graph_capture(steps, False)
        b.set_clusters(1)
        assert b.clusters == (1, 0)
        b.graph_launch(0)
        torch.cuda.synchronize()
        got = [a for r in (0, 1) for l in range(b.n_layers(r)) for a in b.get_grads(r, l)]
        tol = 1e-8 if precision == 64 else 1e-4
        for g, r in zip(got, ref[1]):
            assert _rel(g, r) < tol
    finally:
        b.close()


def test_automatic_choice():
    """What the cases of test_cluster_gpu run as by default: clusters (but for the one
    cube, too small for them), and few heavy envs among many light ones beside single
    CTAs; and where there are none."""
    for sizes, hidden, envs, steps, K, outputs in CASES:
        b = _batch(sizes, hidden, [envs] * len(sizes), steps, K, outputs, 32)
        size, heavy = b.clusters
        b.close()
        assert (size, heavy) == (1, 0) if sizes == (8,) else size > 1 and heavy == envs * len(sizes), sizes
    b = _batch((700, 30), (32, 16), (4, 196), 15, 6, True, 32)
    size, heavy = b.clusters
    assert size > 1 and 1 <= heavy < 200
    b.set_launch_shape(1024, 1)            # no clusters of that many threads
    assert b.clusters == (1, 0)
    b.set_launch_shape(256, 1)
    assert b.clusters[0] > 1
    b.close()
    b = _batch((30,), (16,), (600,), 15, 6, True, 32)
    assert b.clusters == (1, 0)            # more than three envs per SM
    b.close()


def test_refusals_leave_the_choice():
    from cls_b200 import _capi
    b = _batch((93,), (16,), (3,), 9, 9, True, 32)
    try:
        b.set_clusters(4, 2)
        for size, heavy in ((3, 0), (32, 0), (0, 0), (-2, 0), (8, -1)):
            with pytest.raises(_capi.ClsError):
                b.set_clusters(size, heavy)
            assert b.clusters == (4, 2)
        shape = b.launch_shape
        ref = _run(b, 9, False)
        with pytest.raises(_capi.ClsError):
            b.set_launch_shape(1024, 1)    # the clusters asked for do not exist at this size
        assert b.launch_shape == shape and b.clusters == (4, 2)
        _compare(_run(b, 9, False), ref, 32)
        b.set_clusters(-1)
        b.set_launch_shape(1024, 1)
    finally:
        b.close()
