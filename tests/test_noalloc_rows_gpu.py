"""cls_ms_advance_noalloc for robots with hub vertices: rows longer than one thread
takes, against the FP64 restatement of test_zz_no_alloc (its tolerances: FP32 sums
in another order), and without a thread that walks a hub's row alone."""
import ctypes

import numpy as np
import pytest

from helpers import max_rel

pytestmark = pytest.mark.gpu


def _robot(n_v, n_s, hubs, seed):
    """n_s springs in shuffled order: the first vertices have hubs[i] each, on either
    side, the rest connect vertices beyond them."""
    rng = np.random.default_rng(seed)
    a, b = [], []
    for h, deg in enumerate(hubs):
        other = len(hubs) + np.arange(deg) % (n_v - len(hubs))
        side = rng.integers(0, 2, deg).astype(bool)
        a += list(np.where(side, h, other))
        b += list(np.where(side, other, h))
    rest = n_s - len(a)
    lo = len(hubs)
    u = rng.integers(lo, n_v, rest)
    a += list(u)
    b += list(lo + (u - lo + 1 + rng.integers(0, n_v - lo - 1, rest)) % (n_v - lo))
    s = np.zeros((n_s, 5))
    s[:, 0], s[:, 1] = a, b
    s[:, 2], s[:, 3], s[:, 4] = rng.uniform(0.2, 0.5, n_s), rng.uniform(1, 20, n_s), 0.2
    return s[rng.permutation(n_s)]


class _Call:
    def __init__(self, springs, n_v, n_sub, envs, seed=0):
        import torch
        from test_zz_no_alloc import NoallocAdvance, _lib
        rng = np.random.default_rng(seed)
        self.fn = _lib()
        self.x0, self.v0 = rng.uniform(0.0, 1.0, (envs, n_v, 3)), rng.uniform(-0.5, 0.5, (envs, n_v, 3))
        self.act = rng.uniform(-1, 1, (envs, len(springs)))
        self.t = ([torch.tensor(springs[:, c].astype(np.int32), device="cuda:0") for c in (0, 1)] +
                  [torch.tensor(q.copy(), dtype=torch.float32, device="cuda:0")
                   for q in (springs[:, 2], springs[:, 3], springs[:, 4], self.act, self.x0, self.v0)])
        self.ph = (2e-3, -9.8, 0.0, 2.0, 0.1, 0.5)     # dt, gravity, ground, drag, dashpot, friction
        self.args = NoallocAdvance(envs, n_v, len(springs), n_sub, *(q.data_ptr() for q in self.t), *self.ph, None, 0)
        self.stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def __call__(self):
        assert self.fn(ctypes.byref(self.args), self.stream) == 0

    def time(self, n=20, repeats=5):
        """Least time of n calls in a row, per call."""
        import torch
        best = np.inf
        for _ in range(repeats + 1):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for _ in range(n):
                self()
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]) / n)
        return best


@pytest.mark.parametrize("n_v, n_s, hubs, n_sub, envs", [
    (60, 400, (48, 49, 50), 6, 3),             # around the longest row of one thread
    (300, 1000, (299,), 6, 2),
    (300, 1000, (64, 65, 96, 33, 127, 200), 6, 2),
    (900, 4600, (900, 31, 1500, 49), 3, 64),   # near the largest table that fits one CTA
    (40, 700, (70,) * 10, 6, 2),               # every spring on a hub
])
def test_hub_rows(n_v, n_s, hubs, n_sub, envs):
    from test_zz_no_alloc import _advance64
    springs = _robot(n_v, n_s, hubs, n_s)
    call = _Call(springs, n_v, n_sub, envs)
    call()
    dt, g, ground, drag, dash, fric = call.ph
    gx, gv = call.t[6].cpu().numpy(), call.t[7].cpu().numpy()
    for e in range(0, envs, max(1, envs // 3)):
        rx, rv = _advance64(call.x0[e], call.v0[e], springs, call.act[e], n_sub, dt, g, ground, np.exp(-dt * drag),
                            dash, fric)
        assert max_rel(gx[e], rx) < 1e-5
        assert max_rel(gv[e], rv) < 1e-4


def test_a_hub_costs_no_serial_walk():
    """A hub with 900 of 4600 springs: 1.2 times the time of a robot without one (14
    times when one thread sorted and summed its row)."""
    plain = _Call(_robot(900, 4600, (), 1), 900, 32, 64).time()
    hub = _Call(_robot(900, 4600, (900,), 1), 900, 32, 64).time()
    assert hub < 3 * plain


def test_short_calls():
    """One substep of one env: the lists of a robot of 608 springs take no longer than
    the launches of a call that builds none (6500 springs): 0.9 of their time (1.45
    when a vertex's thread sorted its row)."""
    calls = _Call(_robot(93, 608, (), 1), 93, 1, 1), _Call(_robot(900, 6500, (), 1), 900, 1, 1)
    listed, launches = (min(c.time(50) for _ in range(3)) for c in calls)
    assert listed < 1.2 * launches
