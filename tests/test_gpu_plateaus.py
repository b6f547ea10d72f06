"""Pre-smooth on demand of volumes with a plateau: more voxels at one extreme than the lists of candidates hold (a constant
background, a saturated region, a mask, a frame in the face layers), aligned and odd rows.  Against the oracle, and by the
launches of a call against the same volume with noise on its plateau."""
import numpy as np
import pytest
import torch

import nii2mesh_gb300 as n2m
from oracle.oracle import MC33, OLDCUBES, mesh_equal

pytestmark = pytest.mark.gpu
DIMS = [(44, 41, 43), (43, 44, 41)]


class _View:
    def __init__(self, ptr, shape, kind):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (ptr, False), "version": 2, "strides": None}


def _host(ptr, shape, kind):
    return torch.as_tensor(_View(ptr, shape, kind), device="cuda").cpu().numpy()


def _volume(dims, kind, noise=0.0):
    """noise: of the plateau"""
    rng = np.random.default_rng(dims[0])
    nx, ny, nz = dims
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    r = np.sqrt((x - nx / 2) ** 2 + (y - ny / 2) ** 2 + (z - nz / 2) ** 2)
    body = rng.normal(110, 15, (nz, ny, nx))
    flat = rng.normal(0, noise, (nz, ny, nx)) if noise else np.zeros((nz, ny, nx))
    if kind == "background":
        v = np.where(r < 12, body, flat)
    elif kind == "negative":   # padded around a field of view that holds noise
        v = np.where(r < 9, body, np.where(r < 15, rng.normal(-40, 5, r.shape), flat - 3024.0))
    elif kind == "saturated":
        v = np.where(r < 17, 255.0 + flat, rng.normal(5, 3, r.shape))
    elif kind == "mask":
        v = np.where(r < 17, 101.0 + flat, flat)
    elif kind == "frame":      # two layers around, the smallest value nowhere else
        frame = (np.minimum(x, nx - 1 - x) < 2) | (np.minimum(y, ny - 1 - y) < 2) | (np.minimum(z, nz - 1 - z) < 2)
        v = np.where(frame, flat - 70.0, np.where(r < 12, body, rng.normal(-20, 5, r.shape)))
    else:                      # "checker": smoothed to plateaus that no voxel's window holds
        v = np.where(r < 12, body, 2.0 * ((x + y + z) & 1) + flat)
    return v.astype(np.float32)


def _run(v, cubes=n2m.MC33, **o):
    d = torch.from_numpy(v).cuda()
    torch.cuda.synchronize()
    ctx = n2m.Context()
    for _ in range(2):   # the second call has the first one's buffers
        tp, pp, nt, np_, rep = ctx.meshify_device(d.data_ptr(), v.shape[::-1], 54.0, cubes=cubes, **o)
    got = _host(tp, (nt, 3), "<i4"), _host(pp, (np_, 3), "<f8")
    ctx.close()
    return got, rep


@pytest.mark.parametrize("cubes", [n2m.MC33, n2m.OLDCUBES])
@pytest.mark.parametrize("kind", ["background", "negative", "saturated", "mask", "frame", "checker"])
@pytest.mark.parametrize("dims", DIMS)
def test_plateau_values(oracle, dims, kind, cubes):
    v = _volume(dims, kind)
    smooth = oracle.quick_smooth(v.copy())
    for label in (False, True):
        got, rep = _run(v, cubes, only_largest=label, fill_bubbles=label)
        want = oracle.meshify(v, 54.0, OLDCUBES if cubes == n2m.OLDCUBES else MC33, True, label, label)
        ok, d, msg = mesh_equal(got, want, 0.0)
        assert ok, msg
        assert rep["vmin"] == smooth.min() and rep["vmax"] == smooth.max()


@pytest.mark.parametrize("kind", ["background", "negative", "saturated", "mask", "frame"])
@pytest.mark.parametrize("dims", DIMS)
def test_plateau_takes_the_path_of_noise(dims, kind):
    """smoothing again and labelling again are about twenty launches more"""
    o = dict(only_largest=True, fill_bubbles=True)
    flat, noisy = _run(_volume(dims, kind), **o)[1], _run(_volume(dims, kind, 1.0), **o)[1]
    assert abs(flat["kernel_launches"] - noisy["kernel_launches"]) <= 6


@pytest.mark.parametrize("label", [False, True])
@pytest.mark.parametrize("cubes", [n2m.MC33, n2m.OLDCUBES])
@pytest.mark.parametrize("dims", DIMS)
def test_isolevel_on_a_plateau(oracle, dims, cubes, label):
    """a mask meshed at its own value: more undecided voxels than their list holds, so the exact passes run, and the
    report says so"""
    v = (_volume(dims, "mask") > 0).astype(np.float32) * 54.0
    got, rep = _run(v, cubes, only_largest=label, fill_bubbles=label)
    want = oracle.meshify(v, 54.0, OLDCUBES if cubes == n2m.OLDCUBES else MC33, True, label, label)
    ok, d, msg = mesh_equal(got, want, 0.0)
    assert ok, msg
    assert rep["ms_smooth_pass_a"] == 0.0


def test_labelling_waits_for_the_smoothing():
    """half of the volume is a plateau at the isolevel (the approximate smoothing does not hold), half is noise (clusters
    take long): what the labelled call spends before the exact smoothing is done is not another labelling"""
    rng = np.random.default_rng(5)
    v = rng.uniform(0, 108, (160, 192, 196)).astype(np.float32)
    v[:, :, :100] = 54.0
    d = torch.from_numpy(v).cuda()
    torch.cuda.synchronize()
    ctx = n2m.Context()
    ms = {}
    for label in (False, True):
        reps = [ctx.meshify_device(d.data_ptr(), v.shape[::-1], 54.0, only_largest=label, fill_bubbles=label)[4] for _ in range(8)]
        assert all(r["ms_smooth_pass_a"] == 0.0 for r in reps)
        ms[label] = min(r["ms_stage"][0] for r in reps), min(r["ms_stage"][1] for r in reps)
    ctx.close()
    assert ms[True][0] - ms[False][0] < 0.5 * ms[True][1], ms
