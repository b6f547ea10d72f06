"""The degenerate filter looks only at triangles with a vertex close to a grid point: the bound that lets it skip the
others, and meshes full of vertices at, just inside and just outside that distance, against the oracle."""
import itertools

import numpy as np
import pytest

from oracle.oracle import MC33, MC_CLASSIC_TABLE, OLDCUBES, mesh_equal

NEAR = 1.0 / 512


def test_area_bound():
    """three points on three edges of a cube, each at least NEAR from the corners: the area stays above 8 x the
    filter's own 4e-7"""
    g = np.concatenate([[0], np.geomspace(1e-5, 0.5 - NEAR, 14)]) + NEAR
    t = np.concatenate([g, 1 - g])
    edges = []
    for ax in range(3):
        for b in itertools.product((0.0, 1.0), repeat=2):
            p = np.zeros((len(t), 3))
            p[:, [i for i in range(3) if i != ax]] = b
            p[:, ax] = t
            edges.append(p)
    least = min(np.linalg.norm(np.cross(b[None, :, None] - a[:, None, None], c[None, None, :] - a[:, None, None]), axis=-1).min()
                for a, b, c in itertools.combinations(edges, 3)) / 2
    assert least > 8 * 4e-7


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [MC33, MC_CLASSIC_TABLE, OLDCUBES])
@pytest.mark.parametrize("low", [-7.0, -3.2, -2.5])
@pytest.mark.parametrize("dims", [(33, 18, 21), (64, 9, 40)])
def test_values_near_the_isolevel(gpu, oracle, dims, low, variant):
    """edges cut at 10^low .. 1/2 of their length, some exactly at a grid point"""
    rng = np.random.default_rng(int(-low * 10) + dims[0])
    n = dims[::-1]
    v = 64.0 + np.where(rng.random(n) < 0.5, 1, -1) * 32 * 10 ** rng.uniform(low, 0, n)
    v[rng.random(n) < 0.02] = 64.0
    v = v.astype(np.float32)
    got = gpu.meshify(v, 64.0, original_mc=1 if variant == MC_CLASSIC_TABLE else 0, pre_smooth=False, only_largest=False,
                      fill_bubbles=False, oldcubes=variant == OLDCUBES)
    want = oracle.meshify(v, 64.0, variant, False, False, False)
    ok, d, msg = mesh_equal(got, want, 0.0)
    assert ok, msg
