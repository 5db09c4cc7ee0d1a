"""The MPM handle's whole-rollout record: bounded by the caller, and the recomputing
reverse pass that handles without one take, on the same references as the recorded."""
import numpy as np
import pytest

import test_mpm_gpu as recorded
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


@pytest.fixture
def segments(monkeypatch):
    """Handles without a record, counted."""
    from cls_b200 import mpm
    made = []
    real = mpm.MPMBatch

    def make(*a, **k):
        b = real(*a, record_bytes=0, **k)
        assert b.record_bytes == 0
        made.append(b)
        return b

    monkeypatch.setattr(mpm, "MPMBatch", make)
    yield made
    assert made


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("material", ["fixed_corotated", "neo_hookean"])
def test_2d_gradients(segments, material, precision):
    recorded.test_mpm2d_gradients_match_oracle(material, precision)


@pytest.mark.parametrize("precision, tile, order", [(64, 0, "cells"), (32, 0, "cells"), (64, 256, "cells"),
                                                    (32, 48, "cells"), (64, 0, "base_runs"), (32, 0, "base_runs")])
def test_3d(segments, precision, tile, order):
    recorded.test_mpm3d_neo_hookean_fibre_matches_oracle(precision, tile, order)


def test_forward_golden(segments):
    for precision in (64, 32):
        recorded.test_mpm2d_forward_matches_reference_golden(precision)


def test_intervals_and_graph_replay(segments):
    recorded.test_mpm_checkpoint_interval_and_graph_replay()
