"""The MPM handle's whole-rollout record: bounded by the caller."""
import numpy as np
import pytest

from test_mpm_oracle import body3d

pytestmark = pytest.mark.gpu


def _handle(record_bytes, T=60, K=8, n_grid=32, precision=32):
    from cls_b200.mpm import MPMBatch
    pts, musc, fib = body3d(np.random.default_rng(1))
    return MPMBatch(pts, musc, 2, dim=3, fibre=fib, n_muscles=4, max_steps=T, checkpoint_every=K, n_grid=n_grid,
                    bound=3, material="neo_hookean", precision=precision, record_bytes=record_bytes)


@pytest.mark.parametrize("precision", [32, 64])
def test_record_within_the_callers_bound(precision):
    import torch
    from cls_b200 import mpm
    free = lambda: torch.cuda.mem_get_info()[0]
    need = mpm.record_bytes(len(body3d(np.random.default_rng(1))[0]), 3, 32, 60, n_envs=2, precision=precision)
    for bound, want in ((0, 0), (need - 1, 0), (need, need), (None, need)):
        b = _handle(bound, precision=precision)
        assert b.record_bytes == want
        b.close()
    # one segment's records and grids, not the rollout's, without a record
    _handle(0, 2000).close()
    before = free()
    b = _handle(0, 2000, precision=precision)
    assert before - free() < mpm.record_bytes(b.P, 3, 32, 60, n_envs=2, precision=precision)
    b.close()


def test_serving_slot_memory():
    """A slot of the served legged body (1500 steps, K = 50): two segments' records and
    grids, 1.3 GB; 10 GB when every handle took a record of its own accord."""
    import torch
    from cls_b200 import serving, workloads
    mt = workloads.mpm_serving_type()
    serving.MpmSlotBackend(mt, 1, 100, 50, streams=False).close()
    before = torch.cuda.mem_get_info()[0]
    backend = serving.MpmSlotBackend(mt, 1, 1500, 50, streams=False)
    took = before - torch.cuda.mem_get_info()[0]
    backend.close()
    assert took < 2 << 30
