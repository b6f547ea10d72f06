"""HC smoothing's neighbour lists at the valences where their handling changes: lists of 32 entries sort in shared
memory and are paired, longer ones sort in place; repeated indices, single triangles and unused vertices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the kernels work in FP32 on displacements of at most 2 voxels here: ten sweeps of sums that lose 2^-22 each
TOL = 10 * 2 * 2.0 ** -22 * 2


def _fan(n, closed, seed):
    """n triangles around vertex 0, the rim open or closed by a second apex, plus two unused vertices"""
    rng = np.random.default_rng(seed)
    rim = n if closed else n + 1
    a = np.arange(rim) * 2 * np.pi / rim
    p = np.concatenate([[[0, 0, 1.0]], np.stack([np.cos(a), np.sin(a), 0 * a], 1), [[0, 0, -1.0], [5, 5, 5], [6, 5, 5]]])
    t = [(0, 1 + k, 1 + (k + 1) % rim) for k in range(n)]
    if closed:
        t += [(1 + rim, 1 + (k + 1) % rim, 1 + k) for k in range(n)]
    return p + rng.uniform(-0.1, 0.1, p.shape), np.array(t, np.int32)


@pytest.mark.parametrize("lock", [True, False])
@pytest.mark.parametrize("n,closed", [(1, False), (2, False), (6, True), (15, True), (16, True), (16, False), (17, True),
                                      (17, False), (200, True)])
def test_hc_fans(gpu, oracle, n, closed, lock):
    p, t = _fan(n, closed, n)
    got = gpu.laplacian_smoothHC(p, t, 0.1, 0.5, 5, lock)
    want = oracle.laplacian_smoothHC(p, t, 0.1, 0.5, 5, lock)
    assert np.abs(got - want).max() <= TOL


def test_hc_repeated_indices(gpu, oracle):
    p, t = _fan(12, True, 3)
    t = np.concatenate([t, t[:5], [[0, 0, 3], [4, 4, 4], [2, 7, 2]]]).astype(np.int32)   # doubled and collapsed triangles
    got = gpu.laplacian_smoothHC(p, t, 0.1, 0.5, 5, True)
    want = oracle.laplacian_smoothHC(p, t, 0.1, 0.5, 5, True)
    assert np.abs(got - want).max() <= TOL
