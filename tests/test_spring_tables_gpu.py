"""Per-spring tables (each spring evaluated once, one thread sums a vertex) against
the direct gathers of the single-CTA kernels, over vertex degrees around the sizes
of the per-vertex lists: the same terms in the same order, so the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree, n_v", [(1, 2), (7, 9), (8, 200), (16, 60), (17, 60), (24, 90), (25, 90), (41, 60),
                                         (75, 300)])
def test_tables_equal_direct_gathers(degree, n_v):
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch, Robot
    rng = np.random.default_rng(degree)
    x = rng.uniform(0.05, 0.6, (n_v, 3))
    pairs = {(0, j) for j in range(1, min(degree, n_v - 1) + 1)}          # a hub of this degree
    while len(pairs) < min(3 * n_v, n_v * (n_v - 1) // 2) and degree > 1:  # and a sparse rest
        i, j = sorted(rng.integers(1, n_v, 2))
        if i != j:
            pairs.add((int(i), int(j)))
        if n_v < 12:
            break
    springs = np.array([[i, j, np.linalg.norm(x[i] - x[j]), 3e3, 0.2 if k % 3 else 0.0]
                        for k, (i, j) in enumerate(sorted(pairs))])
    robot = Robot.actuated_outputs(x, springs, hidden=[16])
    p = cls_b200.default_params(**workloads._params(13, 5, run_period=3, turn_period=20))
    out = []
    for mode in (0, 1):
        b = MassSpringBatch([robot] * 2, [0, 1], p)
        try:
            b.weights_init(1)
            b.set_spring_tables(mode)
            tv, th = workloads.targets(np.random.default_rng(2), b.T, 2)
            b.set_targets(tv, th)
            b.set_launch_shape(64, 1)       # the reverse pass's table too, whatever the robot's size
            b.simulate(13, per_env=True)
            out.append([b.observables()["center"], *b.final_state(), *b.state_grads(),
                        *(a for l in range(2) for a in b.get_grads(0, l))])
        finally:
            b.close()
    for u, w in zip(*out):
        assert np.isfinite(u).all() and np.array_equal(u, w)
