"""Pre-smooth on demand of volumes whose rows do not begin at multiples of 16 bytes: every remainder of the row length
around a tile's and a lane's columns, volumes that are themselves misaligned, plateaus at the isolevel, values that make the
path give way to the exact passes; against the oracle, which has one way only."""
import numpy as np
import pytest
import torch

import nii2mesh_gb300 as n2m
from oracle.oracle import MC33, OLDCUBES, mesh_equal

pytestmark = pytest.mark.gpu


class _View:
    def __init__(self, ptr, shape, kind):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (ptr, False), "version": 2, "strides": None}


def _host(ptr, shape, kind):
    return torch.as_tensor(_View(ptr, shape, kind), device="cuda").cpu().numpy()


def _check(oracle, v, iso, shift=0, **o):
    n = v.size
    buf = torch.zeros(n + 4, dtype=torch.float32, device="cuda")
    buf[shift:shift + n] = torch.from_numpy(v.ravel()).cuda()
    torch.cuda.synchronize()
    ctx = n2m.Context()
    cubes = o.get("cubes", n2m.MC33)
    want = oracle.meshify(v, iso, OLDCUBES if cubes == n2m.OLDCUBES else MC33, True, o.get("only_largest", False),
                          o.get("fill_bubbles", False))
    assert want is not None
    tp, pp, nt, np_, rep = ctx.meshify_device(buf.data_ptr() + 4 * shift, v.shape[::-1], iso,
                                              **dict(dict(only_largest=False, fill_bubbles=False), **o))
    ok, d, msg = mesh_equal((_host(tp, (nt, 3), "<i4"), _host(pp, (np_, 3), "<f8")), want, 0.0)
    assert ok, msg
    ctx.close()


def _volume(nx, kind):
    rng = np.random.default_rng(nx)
    n = (9, 13, nx)
    if kind == "noise":
        return rng.normal(0, 30, n).astype(np.float32)
    if kind == "plateau":   # smoothed values exactly at the isolevel, extremes repeated
        return np.where(rng.random(n) < 0.5, rng.choice([0.0, 100.0], n), 50.0).astype(np.float32)
    return (rng.normal(0, 30, n) * 10.0 ** rng.integers(-6, 7, n)).astype(np.float32)   # wide range


@pytest.mark.parametrize("cubes", [n2m.MC33, n2m.OLDCUBES])
@pytest.mark.parametrize("kind", ["noise", "plateau", "wide"])
@pytest.mark.parametrize("nx", [5, 6, 7, 9, 33, 62, 63, 65, 66, 67, 69, 127, 130, 131, 193])
def test_row_lengths(oracle, nx, kind, cubes):
    v = _volume(nx, kind)
    iso = 50.0 if kind == "plateau" else 3.0
    _check(oracle, v, iso, cubes=cubes)
    _check(oracle, v, iso, cubes=cubes, only_largest=True, fill_bubbles=True)


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("nx", [8, 61, 64, 68, 128])
def test_misaligned_volume(oracle, nx, shift):
    v = _volume(nx, "noise")
    _check(oracle, v, 3.0, shift)
    _check(oracle, v, 3.0, shift, only_largest=True)
