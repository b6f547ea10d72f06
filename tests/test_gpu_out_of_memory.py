"""A call that the GPU's memory cannot hold fails by itself, and the next call on the same context and thread does not."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_next_call_after_a_failed_allocation(gpu):
    import torch
    ctx = gpu.Context()
    v = np.random.default_rng(2).normal(0, 1, (20, 21, 22)).astype(np.float32)
    want = ctx.meshify(v, 0.5, only_largest=False)
    d = torch.zeros(16, device="cuda")
    torch.cuda.synchronize()
    out, n = C.c_void_p(), C.c_size_t()
    st = gpu.lib().n2m_deflate_device(ctx.h, C.c_void_p(d.data_ptr()), 1 << 45, 0, C.byref(out), C.byref(n))   # before any copy
    assert st == 3, st   # N2M_ERR_OOM
    got = ctx.meshify(v, 0.5, only_largest=False)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
