"""Which bodies one CTA takes whole: never where that is slower than the launches per
substep of a handle without a record (record_bytes = 0), and the largest that it takes
against those."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(dim, P, n_grid, E, record_bytes, precision=32, T=24):
    from cls_b200.mpm import MPMBatch
    rng = np.random.default_rng(P)
    pos = rng.uniform(0.3, 0.6, (P, dim))
    b = MPMBatch(pos, (np.arange(P) % 5 - 1).astype(np.int32), E, dim=dim, n_muscles=4, max_steps=T, n_grid=n_grid,
                 bound=2, material="fixed_corotated" if dim == 2 else "neo_hookean", precision=precision,
                 checkpoint_every=T, dt=1e-4, gravity=-10.0, p_vol=1.0, mu=40.0, la=40.0, act_strength=4.0, mass=1.0,
                 record_bytes=record_bytes)
    b.set_state(np.broadcast_to(pos, (E,) + pos.shape), rng.uniform(-0.3, 0.3, (E,) + pos.shape))
    b.set_actuation(rng.uniform(-1, 1, (T, E, 4)))
    b.set_loss(rng.uniform(0.0, 1.0, T + 1), np.broadcast_to(pos.mean(0) + 0.05, (T + 1, E, dim)),
               rng.uniform(0.5, 1.5, P))
    return b


def _times(b, T=24):
    import torch
    out = []
    for f in (lambda: b.forward(T), lambda: (b.forward(T), b.backward())):
        times = []
        for _ in range(7):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            f()
            ev[1].record()
            torch.cuda.synchronize()
            times.append(ev[0].elapsed_time(ev[1]))
        out.append(np.median(times[2:]))
    return out


@pytest.mark.parametrize("dim, P, n_grid, E", [
    (2, 640, 32, 600), (2, 768, 32, 200), (2, 1200, 32, 200), (2, 200, 64, 600), (2, 2048, 32, 64),
    (3, 64, 12, 600), (3, 200, 12, 600), (3, 300, 12, 1), (3, 640, 12, 1),
])
def test_not_slower_than_launches_per_substep(dim, P, n_grid, E):
    """A forward rollout within the 6 % that its record costs, forward and reverse
    faster (no recompute); 1.1 to 2.7 times as long before the rule looked at the
    dimension, the SMs and what fits beside each other on one."""
    handles = [_batch(dim, P, n_grid, E, r) for r in (None, 0)]
    try:
        (fwd, both), (fwd0, both0) = (_times(b) for b in handles)
    finally:
        for b in handles:
            b.close()
    assert fwd < 1.15 * fwd0 and both < both0


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("dim, P, n_grid, E", [(2, 512, 32, 300), (2, 2048, 32, 148), (3, 512, 12, 148), (3, 256, 12, 99)])
def test_edges_of_the_rule(dim, P, n_grid, E, precision):
    """Bars of the MPM tests (FP64: state 1e-9, loss and gradients 1e-8; FP32: 1e-5, 1e-4)."""
    st, gr = (1e-9, 1e-8) if precision == 64 else (1e-5, 1e-4)
    out = []
    for r in (None, 0):
        b = _batch(dim, P, n_grid, E, r, precision, T=8)
        loss = b.run(8)
        out.append((loss, b.final_state(), b.grads()))
        b.close()
    rel = lambda a, b: float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))
    (l, s, g), (l0, s0, g0) = out
    assert abs(l - l0) <= gr * abs(l0)
    assert rel(s[0], s0[0]) < st and rel(s[1], s0[1]) < (st if precision == 64 else gr)
    for k in g0:
        assert rel(g[k], g0[k]) < gr, k
