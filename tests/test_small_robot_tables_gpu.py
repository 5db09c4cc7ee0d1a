"""Robots of few vertices run the fused forward pass without spring tables by default,
where the direct gather's half-warps are faster than a thread per vertex; the same
bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(n, precision=32, steps=101):
    import cls_b200
    from cls_b200 import robot_design, workloads
    from cls_b200.batch import MassSpringBatch, Robot
    robot = Robot.actuated_outputs(*robot_design.random_lattice(np.random.default_rng(n), n), hidden=[16])
    b = MassSpringBatch([robot], [0], cls_b200.default_params(threads_per_block=256, **workloads._params(
        steps + 2, steps + 4, precision=precision)))
    b.set_controller_path("per_env")
    b.set_clusters(1)
    b.weights_init(1)
    b.set_targets(*workloads.targets(np.random.default_rng(2), b.T, 1))
    return b


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [16, 28, 60])
def test_same_bits(n, precision):
    """Below, at and above 8 vertices per 64 threads; FP64 at 32 vertices."""
    b = _batch(n, precision, 21)
    out = []
    for mode in (-1, 0, 1):
        b.set_spring_tables(mode)
        assert b.spring_tables == (mode != 0)
        b.simulate(21)
        out.append([*b.final_state(), *b.state_grads(), *b.get_grads(0, 0)])
    b.close()
    for other in out[1:]:
        for u, w in zip(out[0], other):
            assert np.isfinite(u).all() and np.array_equal(u, w)


def test_forward_time():
    """101 substeps of one robot of 30 vertices: 0.59 ms, 0.70 with tables."""
    import torch
    b = _batch(30)
    try:
        b.set_stream(torch.cuda.current_stream().cuda_stream)
        times = {}
        for mode in (-1, 1):
            b.set_spring_tables(mode)
            t = []
            for _ in range(15):
                ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                ev[0].record()
                b.forward_eval(101)
                ev[1].record()
                torch.cuda.synchronize()
                t.append(ev[0].elapsed_time(ev[1]))
            times[mode] = np.median(t[3:])
        assert times[-1] < 0.95 * times[1]
    finally:
        b.close()
