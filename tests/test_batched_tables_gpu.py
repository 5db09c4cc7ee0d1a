"""Spring tables of the batched controller's step kernels: reported as they are, on
demand in FP64, and never the reason that a robot is refused."""
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
    """Automatic: FP32 with tables, FP64 without; mode 1 has them in both, with the bits
    of the direct gathers."""
    from cls_b200 import robot_design
    from cls_b200.batch import Robot
    b = _batch(Robot.actuated_outputs(*robot_design.quadruped_lattice(), hidden=[16]), 5, precision)
    try:
        assert b.spring_tables
        b.set_controller_path("batched")
        assert b.spring_tables == (precision == 32)
        out = []
        for mode in (-1, 0, 1):
            b.set_spring_tables(mode)
            assert b.spring_tables == {-1: precision == 32, 0: False, 1: True}[mode]
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
