"""cls_ms_advance_noalloc of large robots in few envs, a cluster of CTAs per env: against
the FP64 restatement of test_zz_no_alloc (its tolerances), around the numbers of springs
and envs where clusters of 8 and of 4 begin and end, with hubs whose springs overflow a
CTA's table; and short calls as fast as launches per phase."""
import numpy as np
import pytest

from helpers import max_rel
from test_noalloc_rows_gpu import _Call, _robot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sub", [1, 3])
@pytest.mark.parametrize("n_v, n_s, hubs, envs", [
    (220, 1299, (), 1), (220, 1300, (), 1), (236, 1378, (), 12), (236, 1378, (), 13), (236, 1378, (), 29),
    (236, 1378, (), 30),
    (900, 4600, (), 3), (1031, 4601, (), 17),    # ragged shares of the vertices
    (900, 4600, (49, 50, 900), 2),               # long rows
    (900, 4600, (4000,), 2),                     # a hub beyond its CTA's table
    (900, 4600, (2400, 2000), 20),               # clusters of 4
    (6, 1500, (1480,), 2),                       # fewer vertices than CTAs
])
def test_clusters(n_v, n_s, hubs, envs, n_sub):
    from test_zz_no_alloc import _advance64
    springs = _robot(n_v, n_s, hubs, n_s)
    call = _Call(springs, n_v, n_sub, envs)
    call()
    dt, g, ground, drag, dash, fric = call.ph
    gx, gv = call.t[6].cpu().numpy(), call.t[7].cpu().numpy()
    for e in sorted({0, envs // 2, envs - 1}):
        rx, rv = _advance64(call.x0[e], call.v0[e], springs, call.act[e], n_sub, dt, g, ground, np.exp(-dt * drag),
                            dash, fric)
        assert max_rel(gx[e], rx) < 1e-5
        assert max_rel(gv[e], rv) < 1e-4


def test_skipped_springs():
    """Springs with an end outside the robot are skipped, as in the other forms."""
    springs = _robot(300, 2000, (), 5)
    extra = springs[:100].copy()
    extra[::2, 0], extra[1::2, 1] = -1, 300
    mixed = np.concatenate([springs, extra])[np.random.default_rng(1).permutation(2100)]
    keep = mixed[(mixed[:, 0] >= 0) & (mixed[:, 1] < 300)]
    a, b = _Call(mixed, 300, 4, 1), _Call(keep, 300, 4, 1)
    b.t[5].copy_(a.t[5][:, [i for i in range(2100) if mixed[i, 0] >= 0 and mixed[i, 1] < 300]])
    for c, o in ((a, a), (b, a)):
        c.t[6].copy_(o.t[6]), c.t[7].copy_(o.t[7])
    x, v = a.t[6].clone(), a.t[7].clone()
    b.t[6].copy_(x), b.t[7].copy_(v)
    a()
    b()
    for k in (6, 7):
        assert np.array_equal(a.t[k].cpu().numpy(), b.t[k].cpu().numpy())


def test_short_calls():
    """One substep of one robot of 4600 springs: as long as a call that builds no lists
    (6500 springs, launches per phase); 1.9 times when one CTA built them."""
    calls = _Call(_robot(900, 4600, (), 1), 900, 1, 1), _Call(_robot(900, 6500, (), 1), 900, 1, 1)
    listed, launches = (min(c.time(50) for _ in range(3)) for c in calls)
    assert listed < 1.35 * launches
