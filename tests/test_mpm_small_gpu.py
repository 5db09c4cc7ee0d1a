"""MPM bodies that one CTA takes whole (default particle order) against the
general kernels (cells order), and rollouts recorded whole against recomputed
segments.  Tolerances: the MPM tests' bars (FP64: state 1e-9, loss and gradients
1e-8; FP32: 1e-5 and 1e-4)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(order, dim, pos, mus, M, E, T, steps, K, precision, n_grid, material, seed):
    from cls_b200 import mpm
    b = mpm.MPMBatch(pos, mus, E, dim=dim, n_muscles=M, max_steps=T, n_grid=n_grid, bound=2, material=material,
                     precision=precision, checkpoint_every=K, dt=1e-3, gravity=-10.0, p_vol=1.0, mu=40.0, la=40.0,
                     act_strength=4.0, mass=1.0, particle_order=order)
    rng = np.random.default_rng(seed)
    try:
        b.set_state(np.broadcast_to(pos, (E,) + pos.shape), rng.uniform(-0.3, 0.3, (E,) + pos.shape))
        b.set_actuation(rng.uniform(-1, 1, (T, E, M)))
        w = rng.uniform(0.0, 1.0, T + 1)
        b.set_loss(w, np.broadcast_to(pos.mean(0) + 0.05, (T + 1, E, dim)), rng.uniform(0.5, 1.5, len(pos)))
        loss = b.run(steps)
        return loss, b.centers()[:steps + 1], b.final_state(), b.grads()
    finally:
        b.close()


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _check(got, ref, precision):
    st, gr = (1e-9, 1e-8) if precision == 64 else (1e-5, 1e-4)
    assert abs(got[0] - ref[0]) <= gr * abs(ref[0])
    assert _rel(got[1], ref[1]) < st
    for g, r in zip(got[2][:2], ref[2][:2]):
        assert _rel(g, r) < (st if precision == 64 else gr)
    for k in ref[3]:
        assert _rel(got[3][k], ref[3][k]) < gr, k


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("dim, P, n_grid, E, steps", [
    (2, 1, 16, 1, 1), (2, 31, 16, 3, 7), (2, 33, 24, 2, 20), (2, 700, 32, 2, 12),
    (2, 896, 32, 1, 6),       # the largest body one CTA takes in a small batch
    (2, 897, 32, 1, 6),       # beyond it: the general kernels in both orders
    (2, 2048, 32, 64, 4),     # the largest in a batch that fills the GPU
    (3, 65, 12, 2, 9), (3, 600, 14, 1, 5),
])
def test_one_cta_per_env(dim, P, n_grid, E, steps, precision):
    rng = np.random.default_rng(P)
    pos = rng.uniform(0.35, 0.65, (P, dim))
    mus = rng.integers(-1, 3, P).astype(np.int32)
    material = "fixed_corotated" if dim == 2 else "neo_hookean"
    args = (dim, pos, mus, 3, E, steps + 3, steps, 4, precision, n_grid, material, P)
    _check(_run("base_runs", *args), _run("cells", *args), precision)


@pytest.mark.parametrize("precision", [32, 64])
def test_whole_record_equals_recomputed_segments(precision):
    """40 steps recorded whole (K = 20: no more slots than two segments) and the
    same body with K = 5 over a rollout too long to record in two segments; a
    record of a sixteenth of the free memory would hold either, so the second
    handle asks for more steps than that."""
    from cls_b200 import workloads
    pos, mus, _ = workloads.legged_body(n_grid=64)
    keep = np.random.default_rng(0).permutation(len(pos))[:4000]
    args = (3, pos[keep], mus[keep], 16, 1)
    whole = _run("base_runs", *args, 40, 40, 20, precision, 64, "neo_hookean", 3)
    import torch
    free = torch.cuda.mem_get_info()[0]
    long_t = int(free / 16 / (64 ** 3 * 4 * (precision // 8))) + 100
    seg = _run_long(args, long_t, precision)
    _check(whole, seg, precision)


def _run_long(args, T, precision):
    """As _run with T steps of room: the same first 40 steps' inputs."""
    from cls_b200 import mpm
    dim, pos, mus, M, E = args
    b = mpm.MPMBatch(pos, mus, E, dim=dim, n_muscles=M, max_steps=T, n_grid=64, bound=2, material="neo_hookean",
                     precision=precision, checkpoint_every=5, dt=1e-3, gravity=-10.0, p_vol=1.0, mu=40.0, la=40.0,
                     act_strength=4.0, mass=1.0, particle_order="base_runs")
    rng = np.random.default_rng(3)
    try:
        b.set_state(np.broadcast_to(pos, (E,) + pos.shape), rng.uniform(-0.3, 0.3, (E,) + pos.shape))
        act = np.zeros((T, E, M))
        act[:40] = rng.uniform(-1, 1, (40, E, M))
        b.set_actuation(act)
        w = np.zeros(T + 1)
        w[:41] = rng.uniform(0.0, 1.0, 41)
        b.set_loss(w, np.broadcast_to(pos.mean(0) + 0.05, (T + 1, E, dim)), rng.uniform(0.5, 1.5, len(pos)))
        loss = b.run(40)
        g = b.grads()
        g["act"] = g["act"][:40]
        return loss, b.centers()[:41], b.final_state(), g
    finally:
        b.close()
