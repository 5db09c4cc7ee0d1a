"""A captured MPM step keeps the loss weights of its capture, whichever kernels run it;
an eager step takes the present ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("P, T", [(100, 12), (100, 700),   # one CTA per env; weights of one launch and of several
                                  (1500, 12)])             # launches per substep
def test_captured_weights(P, T, precision):
    import torch
    from cls_b200.mpm import MPMBatch
    rng = np.random.default_rng(P)
    pos = rng.uniform(0.35, 0.6, (P, 2))
    b = MPMBatch(pos, (np.arange(P) % 3 - 1).astype(np.int32), 1, dim=2, n_muscles=2, max_steps=T, n_grid=32, bound=2,
                 precision=precision, checkpoint_every=T, dt=1e-4)
    b.set_actuation(rng.uniform(-1, 1, (T, 1, 2)))
    first, second = rng.uniform(0.5, 1.0, (2, T + 1))
    target = np.full((T + 1, 1, 2), 0.5)
    grads = lambda: b.grads()["x0"]
    rel = lambda a, c: np.linalg.norm(a - c) / np.linalg.norm(c)
    try:
        b.set_loss(first, target, rng.uniform(0.5, 1.5, P))
        b.run(T)
        want_first = grads()
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        b.graph_capture(T)
        b.set_loss(second)
        b.run(T)
        want_second = grads()
        b.graph_launch()
        replayed = grads()
        b.run(T)
        again = grads()
    finally:
        b.close()
    tol = 1e-9 if precision == 64 else 1e-4        # the MPM tests' gradient bars, with room for the atomics' order
    assert rel(want_second, want_first) > 10 * tol       # else the two weights say nothing
    assert rel(replayed, want_first) < tol
    assert rel(again, want_second) < tol
