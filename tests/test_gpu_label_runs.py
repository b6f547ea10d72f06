"""Labelled meshing and bwlabel where the run kernels change their way: rows of one, 32, 64 and more words, rows that end
inside a word, long winding components, and volumes in which labelling leaves nothing to mask."""
import numpy as np
import pytest

from oracle.oracle import MC33, OLDCUBES, mesh_equal

pytestmark = pytest.mark.gpu


def _noise(shape, seed, level):
    rng = np.random.default_rng(seed)
    v = rng.uniform(0, 40, shape).astype(np.float32)
    v[rng.random(shape) < level] = 100.0
    return v


@pytest.mark.parametrize("variant", [MC33, OLDCUBES])
@pytest.mark.parametrize("smooth,bubbles", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("dims", [(31, 9, 8), (33, 17, 9), (70, 8, 41), (1025, 7, 6), (2049, 6, 6), (2600, 9, 7)])
def test_meshify_rows(gpu, oracle, dims, smooth, bubbles, variant):
    v = _noise(dims[::-1], dims[0], 0.3)
    got = gpu.meshify(v, 50.0, original_mc=0, pre_smooth=smooth, only_largest=True, fill_bubbles=bubbles,
                      oldcubes=variant == OLDCUBES)
    want = oracle.meshify(v, 50.0, variant, smooth, True, bubbles)
    assert (got is None) == (want is None)
    if want is not None:
        ok, d, msg = mesh_equal(got, want, 0.0)
        assert ok, msg


@pytest.mark.parametrize("smooth", [True, False])
@pytest.mark.parametrize("fill", ["one_hole", "iso_at_minimum"])
def test_meshify_nothing_masked(gpu, oracle, fill, smooth):
    """no voxel outside the kept set and its shell; a minimum that is not below iso"""
    v = np.full((12, 11, 37), 100, np.float32)
    v[5, 5, 9] = v[5, 5, 20:24] = 10
    if fill == "iso_at_minimum":
        v[:] = np.where(v < 50, 50, v)
    got = gpu.meshify(v, 50.0, original_mc=0, pre_smooth=smooth, only_largest=True, fill_bubbles=False)
    want = oracle.meshify(v, 50.0, MC33, smooth, True, False)
    assert (got is None) == (want is None)
    if want is not None:
        ok, d, msg = mesh_equal(got, want, 0.0)
        assert ok, msg


@pytest.mark.parametrize("conn", [6, 18, 26])
@pytest.mark.parametrize("largest,bubbles", [(False, False), (True, False), (True, True)])
def test_bwlabel_winding(gpu, oracle, conn, largest, bubbles):
    """a path that winds through every row of a wide volume (links run the whole way), with noise around it"""
    v = np.zeros((9, 33, 67), np.float32)
    for z in range(0, 9, 2):
        for k, y in enumerate(range(0, 33, 2)):
            v[z, y, :] = 1
            if y + 1 < 33:
                v[z, y + 1, 66 if k % 2 else 0] = 1
        if z + 1 < 9:
            v[z + 1, 32 if (z // 2) % 2 == 0 else 0, 66 if (z // 2) % 2 == 0 else 0] = 1
    v[np.random.default_rng(conn).random(v.shape) < 0.02] = 1
    got, gn = gpu.bwlabel(v, conn, largest, bubbles)
    want, wn = oracle.bwlabel(v, conn, largest, bubbles)
    assert gn == wn
    assert np.array_equal(got, want)
