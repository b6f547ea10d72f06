"""The emit takes 8, 16 or 32 active words at a time, by how many there are per resident warp; 32 takes more than a million and
a half of them: rows of a few voxels (one word each) full of small structures, every marching-cubes variant and the batched
atlas.  Smaller volumes of the same kind take 16 and 8."""
import numpy as np
import pytest

from oracle.oracle import MC33, MC_CLASSIC_TABLE, OLDCUBES, mesh_equal

pytestmark = pytest.mark.gpu
WARPS = 152 * 10 * 4   # resident, at most (shared memory)


def _volume(side):
    """(volume, active words of its padded grid: rows with a corner of a mixed cube)"""
    rng = np.random.default_rng(side)
    v = rng.uniform(0, 0.4, (side, side, 7)).astype(np.float32)
    v[rng.random(v.shape) < 0.04] = 1.0
    v[rng.random(v.shape) < 0.005] = 0.6
    row = (v > 0.5).any(2)   # no row is full of them
    row = np.pad(row, ((1, 1), (1, 1)))
    return v, int((row[:-1, :-1] | row[1:, :-1] | row[:-1, 1:] | row[1:, 1:]).sum())


@pytest.mark.parametrize("variant", [MC33, MC_CLASSIC_TABLE, OLDCUBES])
@pytest.mark.parametrize("side,group", [(1500, 32), (600, 16), (120, 8)])
def test_volume(gpu, oracle, side, group, variant):
    v, active = _volume(side)
    assert (active >= 256 * WARPS) if group == 32 else (active < 100 * WARPS if group == 16 else active < 4 * WARPS)
    got = gpu.meshify(v, 0.5, original_mc=1 if variant == MC_CLASSIC_TABLE else 0, pre_smooth=False, only_largest=False,
                      oldcubes=variant == OLDCUBES)
    want = oracle.meshify(v, 0.5, variant, False, False, False)
    ok, d, msg = mesh_equal(got, want, 0.0)
    assert ok, msg


def test_atlas(gpu):
    """three labels, against each of them as a volume of its own"""
    v, active = _volume(1500)
    assert active >= 256 * WARPS
    lab = (v > 0.5).astype(np.int16)
    lab[500:1000] *= 2
    lab[1000:] *= 3
    ctx = gpu.Context()
    o = dict(pre_smooth=False, only_largest=False, fill_bubbles=False, post_smooth=0)
    for label, status, tris, pts in ctx.atlas(lab, **o):
        assert status == 0
        t, p, _ = ctx.meshify((lab == label).astype(np.float32), 0.5, pre_smooth=False, only_largest=False)
        assert np.array_equal(t, tris) and np.array_equal(p, pts)
    ctx.close()
