"""One context from mesh to mesh: the emit and the degenerate filter run with the buffers of earlier calls, and again when
the mesh does not fit; few, many and no weld candidates; isolevels that have to be replaced after the labelling ran."""
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


def _volume(kind, n, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(0, 100, n).astype(np.float32)
    if kind == "lattice":   # values at the isolevel: vertices at grid points, welds
        v = rng.choice([10.0, 50.0, 90.0], n, p=[0.45, 0.1, 0.45]).astype(np.float32)
    if kind == "few":
        v[n[0] // 2, n[1] // 2, :3] = 50.0
    return v


@pytest.mark.parametrize("cubes", [n2m.MC33, n2m.OLDCUBES])
def test_growing_and_shrinking(gpu, oracle, cubes):
    ctx = n2m.Context()
    steps = [("noise", (6, 7, 9)), ("lattice", (20, 21, 22)), ("few", (9, 8, 10)), ("noise", (40, 33, 50)), ("lattice", (5, 6, 7)),
             ("noise", (41, 33, 50)), ("few", (30, 20, 20)), ("lattice", (30, 31, 40))]
    for k, (kind, n) in enumerate(steps):
        for pre, largest, iso in ((False, False, 50.0), (True, True, 50.0), (True, True, 500.0), (False, True, -5.0)):
            v = _volume(kind, n, k)
            d = torch.from_numpy(v).cuda()
            torch.cuda.synchronize()
            want = oracle.meshify(v, iso, OLDCUBES if cubes == n2m.OLDCUBES else MC33, pre, largest, False)
            try:
                tp, pp, nt, np_, rep = ctx.meshify_device(d.data_ptr(), n[::-1], iso, cubes=cubes, pre_smooth=pre,
                                                          only_largest=largest)
            except Exception:
                assert want is None
                continue
            assert want is not None
            ok, dist, msg = mesh_equal((_host(tp, (nt, 3), "<i4"), _host(pp, (np_, 3), "<f8")), want, 0.0)
            assert ok, (k, kind, pre, largest, iso, msg)

