"""Spring tables of the batched controller's step kernels: reported as they are, and
never the reason that a robot is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(robot, envs, precision, threads=0, steps=9):
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch
    b = MassSpringBatch([robot], [0] * envs, cls_b200.default_params(
        threads_per_block=threads, **workloads._params(steps, 4, precision=precision, run_period=3, turn_period=20)))
    b.weights_init(1)
    b.set_targets(*workloads.targets(np.random.default_rng(2), b.T, envs))
    return b


@pytest.mark.parametrize("precision", [32, 64])
def test_report_and_choice(precision):
    """On by default, with the bits of the direct gathers."""
    from cls_b200 import robot_design
    from cls_b200.batch import Robot
    b = _batch(Robot.actuated_outputs(*robot_design.quadruped_lattice(), hidden=[16]), 5, precision)
    try:
        assert b.spring_tables
        b.set_controller_path("batched")
        assert b.spring_tables
        out = []
        for mode in (-1, 0, 1):
            b.set_spring_tables(mode)
            assert b.spring_tables == (mode != 0)
            b.simulate(9)
            out.append([*b.final_state(), *b.state_grads()])
        for other in out[1:]:
            for u, w in zip(out[0], other):
                assert np.isfinite(u).all() and np.array_equal(u, w)
        b.set_controller_path("per_env")
        assert b.spring_tables
    finally:
        b.close()


def _chain(n):
    from cls_b200.batch import Robot
    x = np.stack([0.02 * np.arange(n) % 3.0, 0.2 + 0.05 * (np.arange(n) // 150), 0.02 * (np.arange(n) % 7)], 1)
    s = np.array([[i, i + 1, np.linalg.norm(x[i] - x[i + 1]), 10.0, 0.2 if i < 8 else 0.0] for i in range(n - 1)])
    return Robot.actuated_outputs(x, s, hidden=[8])


def test_largest_robot_of_small_blocks():
    """The largest chains that the fused kernels of 64 threads take, with their tables:
    the batched step kernels, of 256 threads, take them too, without."""
    from cls_b200 import _capi
    lo, hi = 1000, 3000                      # taken, refused
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            _batch(_chain(mid), 2, 32, 64).close()
            lo = mid
        except _capi.ClsError:
            hi = mid
    b = _batch(_chain(lo), 2, 32, 64)
    try:
        assert b.spring_tables
        b.set_controller_path("batched")
        b.simulate(9)
        assert all(np.isfinite(a).all() for a in (*b.final_state(), *b.state_grads()))
    finally:
        b.close()


def test_fp64_robots_beyond_two_per_sm():
    """400 FP64 robots take 1.03 times as long as 256: four step CTAs fit an SM (1.35 when
    two did and launches that waited took their room)."""
    import torch
    from cls_b200 import robot_design
    from cls_b200.batch import Robot
    robot = Robot.actuated_outputs(*robot_design.random_lattice(np.random.default_rng(150), 150), hidden=[64])
    times = []
    for envs in (256, 400):
        b = _batch(robot, envs, 64, steps=22)
        try:
            b.set_controller_path("batched")
            b.set_stream(torch.cuda.current_stream().cuda_stream)
            t = []
            for _ in range(9):
                ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                ev[0].record()
                b.simulate(21)
                ev[1].record()
                torch.cuda.synchronize()
                t.append(ev[0].elapsed_time(ev[1]))
            times.append(np.median(t[2:]))
        finally:
            b.close()
    assert times[1] < 1.2 * times[0]
