"""marchingCubes() of a range without a cube, on a context that holds the buffers of an earlier mesh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [((40, 40, 40), (0, 0, 0)), ((3, 3, 3), (3, 3, 3)), ((2, 2, 2), (9, 3, 9))])
def test_oldcubes_range_without_a_cube(gpu, lo, hi):
    v = np.random.default_rng(1).normal(0, 1, (42, 42, 42)).astype(np.float32)
    whole = gpu.marching_cubes(v, (0, 0, 0), (42, 42, 42), 0.5, oldcubes=True)
    assert whole is not None
    assert gpu.marching_cubes(v, lo, hi, 0.5, oldcubes=True) is None
    assert gpu.lib().n2m_last_error().decode() == "marching cubes produced no surface"
    again = gpu.marching_cubes(v, (0, 0, 0), (42, 42, 42), 0.5, oldcubes=True)
    assert np.array_equal(whole[0], again[0]) and np.array_equal(whole[1], again[1])
