"""cls_ms_advance_noalloc from two host threads: calls with a large and a small
robot, each on its own stream, never fail for one another."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_and_small_robots_from_two_threads():
    import torch
    from test_zz_no_alloc import NoallocAdvance, _lib
    fn = _lib()
    failed = [0, 0]

    def call(k, n_v, n_s):
        stream = torch.cuda.Stream()
        f32 = dict(dtype=torch.float32, device="cuda:0")
        a = np.random.default_rng(k).integers(0, n_v, n_s).astype(np.int32)
        ab = [torch.tensor(t, device="cuda:0") for t in (a, ((a + 1) % n_v).astype(np.int32))]
        params = [torch.rand(n_s, **f32) for _ in range(4)]
        x, v = torch.rand((1, n_v, 3), **f32), torch.zeros((1, n_v, 3), **f32)
        args = NoallocAdvance(1, n_v, n_s, 1, *(t.data_ptr() for t in ab + params + [x, v]), 1e-4, -9.8, 0.0, 2.0,
                              0.1, 0.5, None, 0)
        torch.cuda.synchronize()
        for _ in range(3000):
            failed[k] += fn(ctypes.byref(args), ctypes.c_void_p(stream.cuda_stream)) != 0
        stream.synchronize()

    threads = [threading.Thread(target=call, args=a) for a in ((0, 900, 4600), (1, 300, 1500))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == [0, 0]
