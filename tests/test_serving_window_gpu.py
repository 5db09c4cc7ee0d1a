"""A served request's result is the same to the bit whatever else its windows hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(300,) * 16, (700,) * 2 + (60,) * 150, (40,) * 320])
@pytest.mark.parametrize("precision", [32, 64])
def test_result_alone_and_among_others(sizes, precision):
    import cls_b200
    from cls_b200 import robot_design, workloads
    from cls_b200.batch import MassSpringBatch, Robot
    kinds = {n: Robot.actuated_outputs(*robot_design.random_lattice(np.random.default_rng(n), n), hidden=[32, 16])
             for n in set(sizes)}
    S, T, K = len(sizes), 21, 10
    b = MassSpringBatch([kinds[n] for n in sizes], list(range(S)), cls_b200.default_params(
        **workloads._params(T, K, precision=precision, run_period=5, turn_period=30)))
    b.weights_init(1)
    first = {n: sizes.index(n) for n in set(sizes)}
    for e, n in enumerate(sizes):                  # the slots of a class hold the same controller
        if e != first[n]:
            for l in range(b.n_layers(e)):
                b.set_weights(e, l, *b.get_weights(first[n], l))
    tv, th = np.zeros((T, 3)), np.full(T, 0.03)
    tv[:, 0] = 0.05

    def serve(slot, others):
        """Loss, final state and gradients of the request on `slot`."""
        active = [slot, *others]
        for e in active:
            b.serve_reset_env(e, kinds[sizes[e]].objects, None, tv * (1.0 if e == slot else 0.4), th)
        steps = np.full(S, 2, np.int32)
        steps[active] = T
        win = np.zeros((S, 4), np.int32)
        for t0 in (0, K):
            win[active] = (t0, t0 + K, t0 // K, 0)
            b.serve_forward(win, steps)
        only = np.zeros(S, np.int32)
        only[active] = T
        loss = b.serve_loss(only)[:, slot]
        for seg in (1, 0):
            win[active] = (seg * K, seg * K + K, seg, seg == 1)
            b.serve_backward(win, steps)
        return [loss, *b.serve_env_state(slot), *(a for l in range(b.n_layers(slot)) for a in b.get_grads(slot, l))]

    try:
        for n in set(sizes):
            alone = serve(first[n], [])
            last = S - 1 - sizes[::-1].index(n)    # another slot of the class, among all the others
            rest = [e for e in range(S) if e != last]
            for others in (rest[:3], rest):
                got = serve(last, others)
                assert np.any(alone[-2] != 0)
                assert all(np.array_equal(g, a) for g, a in zip(got, alone)), (n, len(others))
    finally:
        b.close()
