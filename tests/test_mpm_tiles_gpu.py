"""MPM handles with warp tiles of different sizes, and without, beside each other in one
process: a later handle takes nothing from an earlier one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(tile, precision=32):
    from cls_b200.mpm import MPMBatch
    rng = np.random.default_rng(1)
    pos = rng.uniform(0.4, 0.6, (600, 3))
    b = MPMBatch(pos, (np.arange(600) % 3 - 1).astype(np.int32), 1, dim=3, n_muscles=2, max_steps=6, n_grid=32, bound=3,
                 precision=precision, checkpoint_every=3, dt=1e-4, material="neo_hookean", tile_nodes=tile, record_bytes=0,
                 particle_order=0)          # by cells, which tiles need
    b.set_actuation(rng.uniform(-1, 1, (6, 1, 2)))
    b.set_loss(rng.uniform(0.5, 1.0, 7), np.full((7, 1, 3), 0.5), np.ones(600))
    return b


@pytest.mark.parametrize("later", [64, 0])
@pytest.mark.parametrize("precision", [32, 64])
def test_a_smaller_handle_made_later(later, precision):
    first = _batch(512, precision)
    try:
        want = first.run(6)
        second = _batch(later, precision)
        second.run(6)
        got = first.run(6)
        second.close()
    finally:
        first.close()
    assert np.isfinite(want) and abs(got - want) <= (1e-12 if precision == 64 else 1e-5) * abs(want)
