"""Raw volumes without pre-smoothing: range, bbox and non-finite count are taken slab by slab while the volume arrives, and
the labelling works on the upload itself.  Fewer slices than slabs, as many, more; the isolevel in and out of range; after
each one a smoothed volume and one in device memory on the same context, which must not find the raw one's statistics."""
import numpy as np
import pytest

import nii2mesh_gb300 as n2m
from oracle.oracle import MC33, OLDCUBES, cast_voxels, mesh_equal

pytestmark = pytest.mark.gpu


def _raw(nz, dtype):
    rng = np.random.default_rng(nz)
    n = (nz, 23, 30)
    v = np.where(rng.random(n) < 0.3, rng.normal(150, 20, n), rng.normal(40, 20, n))
    v[rng.random(n) < 0.01] = 400
    if np.issubdtype(dtype, np.integer):
        i = np.iinfo(dtype)
        v = v.round().clip(max(i.min, -500), min(i.max, 500))
    return v.astype(dtype)


def _same(oracle, got, f, iso, cubes, pre, label, fill):
    want = oracle.meshify(f, iso, OLDCUBES if cubes == n2m.OLDCUBES else MC33, pre, label, fill)
    ok, d, msg = mesh_equal(got, want, 0.0)
    assert ok, msg


@pytest.mark.parametrize("label,fill", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("cubes", [n2m.MC33, n2m.OLDCUBES])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32])
@pytest.mark.parametrize("nz", [5, 16, 37])
def test_unsmoothed(oracle, nz, dtype, cubes, label, fill):
    import torch
    raw = _raw(nz, dtype)
    f = cast_voxels(raw, 0.5, -20.0)
    d = torch.from_numpy(f.copy()).cuda()
    torch.cuda.synchronize()
    ctx = n2m.Context()
    o = dict(cubes=cubes, only_largest=label, fill_bubbles=fill)
    for iso in (28.0, 1e6, -1e6):   # the last two are replaced
        t, p, rep = ctx.meshify_typed(raw, 0.5, -20.0, iso, pre_smooth=False, **o)
        _same(oracle, (t, p), f, iso, cubes, False, label, fill)
        assert rep["vmin"] == f.min() and rep["vmax"] == f.max()
    t, p, _ = ctx.meshify(f + 3, 31.0, pre_smooth=True, **o)
    _same(oracle, (t, p), f + 3, 31.0, cubes, True, label, fill)
    ctx.meshify_typed(raw, 0.5, -20.0, 28.0, pre_smooth=False, **o)
    t, p, _ = ctx.meshify(2 * f, 50.0, pre_smooth=False, **o)
    _same(oracle, (t, p), 2 * f, 50.0, cubes, False, label, fill)
    ctx.meshify_typed(raw, 0.5, -20.0, 28.0, pre_smooth=False, **o)
    tp, pp, nt, np_, rep = ctx.meshify_device(d.data_ptr(), f.shape[::-1], 28.0, pre_smooth=False, **o)
    want = oracle.meshify(f, 28.0, OLDCUBES if cubes == n2m.OLDCUBES else MC33, False, label, fill)
    assert (nt, np_) == (len(want[0]), len(want[1])) and rep["vmin"] == f.min() and rep["vmax"] == f.max()
    assert np.array_equal(d.cpu().numpy(), f)   # the caller's volume is as it was
    ctx.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("z", [0, 20, 36])
def test_refused_volumes(oracle, bad, z):
    raw = _raw(37, np.float32)
    ctx = n2m.Context()
    ill = raw.copy()
    ill[z, 5, 7] = bad
    for v in (ill, np.full_like(raw, 7)):   # not finite; no variability
        with pytest.raises(n2m.N2MError):
            ctx.meshify_typed(v, 1.0, 0.0, 95.0, pre_smooth=False)
        t, p, _ = ctx.meshify_typed(raw, 1.0, 0.0, 95.0, pre_smooth=False)
        _same(oracle, (t, p), cast_voxels(raw, 1.0, 0.0), 95.0, n2m.MC33, False, True, False)
    ctx.close()
