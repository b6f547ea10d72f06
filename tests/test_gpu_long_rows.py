"""Vertices far along x, where a stored coordinate is rounded to a 256th of a voxel or worse: whether a vertex counts as close
to a grid point (and its triangles go through the degenerate filter) is decided on the stored coordinate."""
import numpy as np
import pytest

from oracle.oracle import MC33, MC_CLASSIC_TABLE, OLDCUBES, mesh_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [MC33, MC_CLASSIC_TABLE, OLDCUBES])
@pytest.mark.parametrize("nx", [32767])   # the reference's dimensions are short
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_values_near_the_isolevel(gpu, oracle, axis, nx, variant):
    rng = np.random.default_rng(nx + axis)
    n = [7, 6, 5]
    n[2 - axis] = nx
    v = 64.0 + np.where(rng.random(n) < 0.5, 1, -1) * 32 * 10 ** rng.uniform(-5, 0, n)
    v[rng.random(n) < 0.02] = 64.0
    v = v.astype(np.float32)
    got = gpu.meshify(v, 64.0, original_mc=1 if variant == MC_CLASSIC_TABLE else 0, pre_smooth=False, only_largest=False,
                      fill_bubbles=False, oldcubes=variant == OLDCUBES)
    want = oracle.meshify(v, 64.0, variant, False, False, False)
    ok, d, msg = mesh_equal(got, want, 0.0)
    assert ok, msg
