"""MPM serving slots: what the footprint counts is what a slot keeps."""
import numpy as np
import pytest


def _type(**solver):
    from cls_b200.serving import MpmType
    pos = np.random.default_rng(0).uniform(0.4, 0.6, (500, 3))
    return MpmType(pos, np.zeros(500, np.int32), None, n_muscles=2, solver=dict(n_grid=32, **solver))


@pytest.mark.parametrize("dim, n_grid", [(2, 32), (2, 33), (3, 32), (3, 30)])
def test_record_bytes(dim, n_grid):
    """x, v, C and F of a particle and 4 values per node of whole blocks, every step."""
    from cls_b200 import mpm
    side = 8 if dim == 2 else 4
    blocks = ((n_grid + side - 1) // side) ** dim
    want = 7 * 3 * 8 * (500 * (2 * dim + 2 * dim * dim) + 4 * blocks * side ** dim)
    assert mpm.record_bytes(500, dim, n_grid, 7, n_envs=3, precision=64) == want


def test_slots_record_only_what_the_footprint_counts(monkeypatch):
    from cls_b200 import mpm, serving
    made = []

    class Fake:
        class params:
            dt = 1e-4

        def __init__(self, *a, record_bytes=None, **k):
            made.append(record_bytes)

    monkeypatch.setattr(mpm, "MPMBatch", Fake)
    T, K = 1500, 50
    whole = mpm.record_bytes(500, 3, 32, T)
    plain, recorded = _type(), _type(record_bytes=whole)
    for t in (plain, recorded, _type(record_bytes=whole - 1)):
        serving.MpmSlotBackend(t, 2, T, K, streams=False)
    assert made == [0, 0, whole, whole, whole - 1, whole - 1]     # never the library's own bound
    segments = serving.mpm_footprint_bytes(plain, T, K)
    assert segments < whole <= serving.mpm_footprint_bytes(recorded, T, K)
    assert serving.mpm_footprint_bytes(_type(record_bytes=whole - 1), T, K) == segments
