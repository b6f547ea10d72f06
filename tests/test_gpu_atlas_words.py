"""Batched atlas meshing where its word kernels change their way: rows that end inside a word and of several words, a
label that fills the volume, labels in one slice or at a corner, volumes too small to smooth, more labels than a block's
table of boxes holds, negative labels."""
import numpy as np
import pytest

from oracle.oracle import mesh_equal

pytestmark = pytest.mark.gpu


def _check(gpu, oracle, lab, labels=None, **kw):
    ctx = gpu.Context(0)
    batched = ctx.atlas(lab, mode=gpu.ATLAS_BATCHED, post_smooth=0, **kw)
    assert [m[0] for m in batched] == sorted(v for v in np.unique(lab) if v > 0)
    img = lab.astype(np.float32)
    for l, st, t, p in batched:
        if labels is not None and l not in labels:
            continue
        binimg, _ = oracle.binarize_label(img, int(l))
        want = oracle.meshify(binimg, 0.5, 0, kw["pre_smooth"], kw["only_largest"], kw["fill_bubbles"])
        assert (want is None) == bool(st), l
        if not st:
            ok, d, msg = mesh_equal((t, p), want, 0.0)
            assert ok, f"label {l}: {msg}"
    ctx.close()


@pytest.mark.parametrize("largest,bubbles", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("smooth", [True, False])
@pytest.mark.parametrize("dims", [(31, 12, 9), (33, 9, 14), (70, 20, 11), (131, 9, 9), (40, 4, 6), (6, 3, 5)])
def test_noise(gpu, oracle, dims, smooth, largest, bubbles):
    rng = np.random.default_rng(dims[0])
    lab = rng.choice(np.array([0, 1, 2, 7, -3], np.int16), dims[::-1], p=[0.3, 0.4, 0.1, 0.1, 0.1])
    _check(gpu, oracle, lab, pre_smooth=smooth, only_largest=largest, fill_bubbles=bubbles)


@pytest.mark.parametrize("largest,bubbles", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("smooth", [True, False])
def test_whole_volume_slice_and_corner(gpu, oracle, smooth, largest, bubbles):
    lab = np.ones((11, 13, 37), np.int16)
    lab[5, 6, 10:13] = 0          # a bubble in a label that reaches every face
    lab[3, :, :] = 2
    lab[0, 0, 0] = lab[-1, -1, -1] = 3
    _check(gpu, oracle, lab, pre_smooth=smooth, only_largest=largest, fill_bubbles=bubbles)
    full = np.full((8, 9, 35), 5, np.int16)
    full[4, 4, 7] = full[4, 4, 33] = 0
    _check(gpu, oracle, full, pre_smooth=smooth, only_largest=largest, fill_bubbles=bubbles)


def test_many_labels(gpu, oracle):
    """600 labels in short runs: more than a block's table holds, several per thread"""
    rng = np.random.default_rng(4)
    lab = (rng.integers(0, 600, (14, 16, 24)) * (rng.random((14, 16, 24)) < 0.7)).astype(np.int16)
    lab[2:6, 3:7, 3:9] = 32767
    _check(gpu, oracle, lab, labels={1, 17, 255, 256, 599, 32767}, pre_smooth=True, only_largest=True, fill_bubbles=True)
