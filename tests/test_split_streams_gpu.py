"""A launch of the heaviest envs on clusters beside the others on single CTAs: the CTAs that
are out of work leave their SMs to other streams while the heavy envs still run, and
what follows on the stream still waits for these."""
import numpy as np
import pytest

from test_cluster_gpu import _lattice

pytestmark = pytest.mark.gpu


def _batch(sizes, envs, steps):
    import cls_b200
    from cls_b200 import workloads
    from cls_b200.batch import MassSpringBatch
    import torch
    b = MassSpringBatch([_lattice(n, (16,), seed=n) for n in sizes], [r for r, n in enumerate(envs) for _ in range(n)],
                        cls_b200.default_params(**workloads._params(steps + 2, steps + 2, loss=("velocity",))))
    b.set_controller_path("per_env")
    b.weights_init(1)
    b.set_targets(*workloads.targets(np.random.default_rng(2), b.T, b.n_envs))
    stream = torch.cuda.Stream()
    b.set_stream(stream.cuda_stream)
    return b, stream


@pytest.mark.parametrize("reverse", [False, True])
def test_finished_ctas_leave(reverse):
    """One robot of 1200 vertices on a cluster of 2 (several times as long as the 146
    others take): 146 envs on another stream, submitted right behind, finish before it."""
    import torch
    steps = 200
    a, sa = _batch((1200, 30), (1, 146), steps)
    c, sc = _batch((30,), (146,), steps)
    try:
        a.set_clusters(2, 1)
        assert a.clusters == (2, 1)
        ran = []
        for _ in range(3):
            start, end_a, end_c = (torch.cuda.Event(enable_timing=True) for _ in range(3))
            for b in (a, c):
                b.forward(steps)
                b.loss()
            torch.cuda.synchronize()
            start.record(sa)
            sc.wait_event(start)
            for b, s, end in ((a, sa, end_a), (c, sc, end_c)):
                b.backward() if reverse else b.forward(steps)
                end.record(s)
            torch.cuda.synchronize()
            ran.append((start.elapsed_time(end_a), start.elapsed_time(end_c)))
        alone = []
        for _ in range(3):
            start, end_c = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record(sc)
            c.backward() if reverse else c.forward(steps)
            end_c.record(sc)
            torch.cuda.synchronize()
            alone.append(start.elapsed_time(end_c))
        heavy, other = np.median(ran, axis=0)
        assert heavy > 3 * np.median(alone)              # else the envs beside it say nothing
        assert other < 0.9 * heavy
    finally:
        a.close()
        c.close()


def test_the_stream_waits_for_the_heavy_envs():
    """The final state read right behind the launch is that of per-env launches."""
    steps = 60
    b, _ = _batch((1200, 30), (1, 146), steps)
    try:
        b.simulate(steps, per_env=True)
        want = b.final_state()
        b.set_clusters(2, 1)
        for _ in range(5):
            b.forward(steps)
            assert all(np.array_equal(g, w) for g, w in zip(b.final_state(), want))
    finally:
        b.close()
