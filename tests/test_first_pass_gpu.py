"""The first pass of a new handle takes what its later passes take, and handles made
and closed on several threads keep their results apart."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _eval_batch(seed, envs=1, steps=60):
    import cls_b200
    from cls_b200 import robot_design, workloads
    from cls_b200.batch import MassSpringBatch, Robot
    robot = Robot.actuated_outputs(*robot_design.quadruped_lattice(), hidden=[64])
    b = MassSpringBatch([robot], [0] * envs, cls_b200.default_params(**workloads._params(steps + 2, steps)))
    b.weights_init(seed)
    b.set_targets(*workloads.targets(np.random.default_rng(seed), steps + 2, envs))
    return b


def _pass(b, steps=60):
    b.forward_eval(steps)
    return b.observables()["center"], *b.final_state()


def test_first_pass_of_a_new_handle():
    """Median over eight handles: 1.0 of the second pass's time; 4 when the first
    results of a handle allocated page-locked memory."""
    import torch
    first, second = [], []
    for k in range(9):
        b = _eval_batch(k)
        times = []
        for _ in range(2):
            torch.cuda.synchronize()
            t = time.perf_counter()
            _pass(b)
            times.append(time.perf_counter() - t)
        b.close()
        if k:        # the process's first handle loads the kernels
            first.append(times[0])
            second.append(times[1])
    assert np.median(first) < 2 * np.median(second)


def test_handles_on_threads_keep_their_results():
    want = {}
    for k in range(3):
        b = _eval_batch(k, 1 + k)
        want[k] = _pass(b)
        b.close()
    wrong = []

    def work(k):
        import torch
        torch.cuda.set_device(0)
        for _ in range(12):
            b = _eval_batch(k, 1 + k)
            b.set_stream(torch.cuda.Stream().cuda_stream)
            for _ in range(3):
                if not all(np.array_equal(g, r) for g, r in zip(_pass(b), want[k])):
                    wrong.append(k)
            b.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
