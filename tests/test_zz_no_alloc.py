"""cls_ms_advance_noalloc: the entry point for callers that may not allocate
device memory (they cannot create a cls_sim, whose buffers come from
cudaMalloc).  It must reproduce the regular entry point's trajectory while
allocating nothing, on two calls in a row that share its fixed scratch array.

The regular path is cls_forward with a controller whose weights are all zero,
so every spring's actuation is the constant sin(bias); the no-alloc call is
given exactly those actuations.  Tolerances: FP32 positions rel 1e-5 (the
spring sums are accumulated in a different order); velocities rel 1e-4 (the
same rounding, divided by the time step, weighs more against their size)."""
import ctypes

import numpy as np
import pytest

from helpers import batch_from_golden, load_golden, max_rel

pytestmark = pytest.mark.gpu


class NoallocAdvance(ctypes.Structure):
    _fields_ = [("n_envs", ctypes.c_int32), ("n_vertices", ctypes.c_int32),
                ("n_springs", ctypes.c_int32), ("n_substeps", ctypes.c_int32),
                ("spring_a", ctypes.c_void_p), ("spring_b", ctypes.c_void_p),
                ("rest_length", ctypes.c_void_p), ("stiffness", ctypes.c_void_p),
                ("actuation_coef", ctypes.c_void_p), ("actuation", ctypes.c_void_p),
                ("x", ctypes.c_void_p), ("v", ctypes.c_void_p),
                ("dt", ctypes.c_float), ("gravity", ctypes.c_float),
                ("ground_height", ctypes.c_float), ("drag_damping", ctypes.c_float),
                ("dashpot_damping", ctypes.c_float), ("friction", ctypes.c_float),
                ("error_message", ctypes.c_char_p), ("error_capacity", ctypes.c_int32)]


def _lib():
    import cls_b200
    lib = cls_b200._capi.load()
    fn = lib.cls_ms_advance_noalloc
    fn.argtypes = [ctypes.POINTER(NoallocAdvance), ctypes.c_void_p]
    fn.restype = ctypes.c_int32
    return fn


def _reference_final_states(g, n, biases):
    """(x, v) after n and 2n substeps through the regular entry point."""
    out = []
    for steps in (n, 2 * n):
        b = batch_from_golden(g, precision=32, K=8)
        W0, _ = b.get_weights(0, 0)
        W1, _ = b.get_weights(0, 1)
        b.set_weights(0, 0, np.zeros_like(W0), np.zeros(W0.shape[0]))
        b.set_weights(0, 1, np.zeros_like(W1), biases)
        b.forward(steps + 1)            # training rollout: steps substeps
        out.append(b.final_state())
        b.close()
    return out


def test_noalloc_matches_regular_entry_point_twice():
    import torch
    fn = _lib()
    g = load_golden("quad_ref")
    B, N = int(g["B"]), g["objects"].shape[0]
    springs = g["springs"]
    S = springs.shape[0]
    n = 20
    rng = np.random.default_rng(4)
    biases = rng.uniform(-1.0, 1.0, S)
    ref1, ref2 = _reference_final_states(g, n, biases)

    dev = torch.device("cuda:0")
    f32 = dict(dtype=torch.float32, device=dev)
    sa = torch.tensor(springs[:, 0].astype(np.int32), device=dev)
    sb = torch.tensor(springs[:, 1].astype(np.int32), device=dev)
    rest = torch.tensor(springs[:, 2], **f32)
    stiff = torch.tensor(springs[:, 3] * 0.1, **f32)      # the reference's /10
    coef = torch.tensor(springs[:, 4], **f32)
    act = torch.tensor(np.broadcast_to(np.sin(biases.astype(np.float32)), (B, S)).copy(), **f32)
    x = torch.tensor(g["x0"].reshape(B, N, 3), **f32).contiguous()
    v = torch.zeros((B, N, 3), **f32)
    msg = ctypes.create_string_buffer(256)
    a = NoallocAdvance(B, N, S, n, sa.data_ptr(), sb.data_ptr(), rest.data_ptr(), stiff.data_ptr(),
                       coef.data_ptr(), act.data_ptr(), x.data_ptr(), v.data_ptr(),
                       float(g["dt"]), float(g["gravity"]), float(g["ground"]), float(g["drag"]),
                       float(g["dashpot"]), 0.4, ctypes.cast(msg, ctypes.c_char_p), 256)
    stream = torch.cuda.current_stream().cuda_stream
    for call, (rx, rv) in enumerate((ref1, ref2)):   # two calls in a row, continuing the state
        torch.cuda.synchronize()
        free_before = torch.cuda.mem_get_info()[0]
        rc = fn(ctypes.byref(a), ctypes.c_void_p(stream))
        assert rc == 0, msg.value
        torch.cuda.synchronize()
        if call == 1:
            # the first call may load the library's kernels (lazy module
            # loading takes device memory once); the second must take none
            assert torch.cuda.mem_get_info()[0] == free_before
        assert max_rel(x.cpu().numpy().reshape(-1, 3), rx) < 1e-5
        assert max_rel(v.cpu().numpy().reshape(-1, 3), rv) < 1e-4


def test_noalloc_rejects_sizes_beyond_its_scratch():
    import torch
    fn = _lib()
    msg = ctypes.create_string_buffer(256)
    dummy = torch.zeros(16, dtype=torch.float32, device="cuda:0")
    p = dummy.data_ptr()
    a = NoallocAdvance(4096, 1000, 0, 1, None, None, None, None, None, None, p, p,
                       1e-3, -9.8, 0.0, 0.0, 0.1, 0.4, ctypes.cast(msg, ctypes.c_char_p), 256)
    assert fn(ctypes.byref(a), None) == -1
    assert b"exceeds the fixed scratch" in msg.value


def _advance64(x, v, springs, act, n, dt, gravity, ground, drag_s, dashpot, friction):
    """FP64 restatement of one env's substeps (solver_mass_spring.py:86-148)."""
    a, b = springs[:, 0].astype(int), springs[:, 1].astype(int)
    ok = (a >= 0) & (a < len(x)) & (b >= 0) & (b < len(x))
    a, b, l0, k, coef, act = a[ok], b[ok], springs[ok, 2], springs[ok, 3], springs[ok, 4], act[ok]
    for _ in range(n):
        d, dv = x[a] - x[b], v[a] - v[b]
        n2 = (d * d).sum(1)
        length = np.sqrt(n2 + 1e-8) + 1e-4
        nrm = d / np.sqrt(n2)[:, None]
        imp = (dt * (length - l0 * (1 + coef * act)) * k / length)[:, None] * d
        imp += (dashpot * (dv * nrm).sum(1))[:, None] * nrm
        vinc = np.zeros_like(v)
        np.add.at(vinc, a, -imp)
        np.add.at(vinc, b, imp)
        ov = drag_s * v + vinc
        ov[:, 1] += dt * gravity
        hit = (x[:, 1] + dt * ov[:, 1] < ground) & (ov[:, 1] < -1e-4)
        toi = np.where(hit, -(x[:, 1] - ground) / np.where(hit, ov[:, 1], -1.0), 0.0)
        f = np.where(hit, -friction * ov[:, 1], 0.0)
        nv = ov.copy()
        nv[hit, 1] = 0.0
        for c in (0, 2):
            nv[:, c] = np.where(ov[:, c] < 0, np.minimum(0.0, ov[:, c] + f), np.maximum(0.0, ov[:, c] - f))
        x = x + toi[:, None] * ov + (dt - toi)[:, None] * nv
        v = nv
    return x, v


@pytest.mark.parametrize("n_v, n_s, n_sub, envs", [
    (1, 0, 3, 2),            # no springs
    (2, 1, 1, 1), (33, 31, 5, 3), (300, 257, 4, 2), (257, 1025, 7, 2),
    (900, 4600, 3, 2),       # near the largest table that fits one CTA
    (900, 6500, 3, 2),       # beyond it: a launch per phase
    (40, 90, 0, 1),          # nothing to do
])
def test_noalloc_advance_sizes(n_v, n_s, n_sub, envs):
    """One launch per call (springs in shared memory) and one per phase, against
    the FP64 restatement; some springs name vertices that do not exist and are
    skipped.  The file's tolerances."""
    import torch
    fn = _lib()
    rng = np.random.default_rng(n_v + n_s)
    x0 = rng.uniform(0.0, 1.0, (envs, n_v, 3))
    v0 = rng.uniform(-0.5, 0.5, (envs, n_v, 3))
    springs = np.zeros((n_s, 5))
    if n_s:
        a = rng.integers(0, n_v, n_s)
        springs[:, 0], springs[:, 1] = a, (a + 1 + rng.integers(0, max(1, n_v - 1), n_s)) % n_v
        springs[:, 2], springs[:, 3], springs[:, 4] = rng.uniform(0.2, 0.5, n_s), rng.uniform(1, 20, n_s), 0.2
        springs[::7, rng.integers(0, 2)] = n_v + 3
        springs[3::11, 0] = -1
    act = rng.uniform(-1, 1, (envs, n_s))
    ph = dict(dt=2e-3, gravity=-9.8, ground=0.0, drag=2.0, dashpot=0.1, friction=0.5)
    f32 = dict(dtype=torch.float32, device="cuda:0")
    i32 = dict(dtype=torch.int32, device="cuda:0")
    sa, sb = (torch.tensor(springs[:, c].astype(np.int32), **i32) for c in (0, 1))
    rest, stiff, coef = (torch.tensor(springs[:, c].copy(), **f32) for c in (2, 3, 4))
    ta, x, v = torch.tensor(act, **f32), torch.tensor(x0, **f32), torch.tensor(v0, **f32)
    args = NoallocAdvance(envs, n_v, n_s, n_sub, sa.data_ptr(), sb.data_ptr(), rest.data_ptr(), stiff.data_ptr(),
                          coef.data_ptr(), ta.data_ptr(), x.data_ptr(), v.data_ptr(), ph["dt"], ph["gravity"],
                          ph["ground"], ph["drag"], ph["dashpot"], ph["friction"], None, 0)
    assert fn(ctypes.byref(args), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    gx, gv = x.cpu().numpy(), v.cpu().numpy()
    for e in range(envs):
        rx, rv = _advance64(x0[e], v0[e], springs, act[e], n_sub, ph["dt"], ph["gravity"], ph["ground"],
                            np.exp(-ph["dt"] * ph["drag"]), ph["dashpot"], ph["friction"])
        assert max_rel(gx[e], rx) < 1e-5
        assert max_rel(gv[e], rv) < 1e-4
