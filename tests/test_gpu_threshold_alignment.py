"""setThreshold of volumes in device memory that begin at any multiple of 4 bytes, of lengths that are no multiple of 4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 99, 130, 4097, 150001, 1000003])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_misaligned(gpu, oracle, n, shift):
    import torch
    rng = np.random.default_rng(n + shift)
    v = np.where(rng.random(n) < 0.4, rng.normal(100, 15, n), np.where(rng.random(n) < 0.5, 0, rng.normal(20, 9, n)))
    v = v.astype(np.float32)
    if n > 1000:
        v[::97] = np.nan
    d = torch.full((n + 8,), 1e9, device="cuda")   # the voxels around are not the volume's
    d[shift:shift + n] = torch.from_numpy(v).cuda()
    torch.cuda.synchronize()
    ctx = gpu.Context()
    for mode in (1, 2, 3):
        assert ctx.set_threshold_device(d.data_ptr() + 4 * shift, n, mode) == oracle.set_threshold(v, mode), mode
    ctx.close()
