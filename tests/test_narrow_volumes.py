"""Volumes whose rows are one word (at most 30 voxels): boxes of the resident
kernel (begputhinning_b200/csrc/resident.cu) cut along y, along z and along
both, and boxes with more non-empty words than their lists hold, against the
oracle."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.helpers import blobs3d

pytestmark = pytest.mark.gpu


def _thin(ctx, v, grid=0):
    import torch
    from begputhinning_b200 import Batch
    b = Batch(ctx)
    i = b.add(v.shape)
    if grid:
        b.set_grid(grid)
    b.finalize()
    t = torch.from_numpy(v).cuda()
    o = torch.full_like(t, 7)
    b.set_io(i, t, o)
    b.run()
    got, plan, stat = o.cpu().numpy(), b.plan(i), b.stats(i)
    b.close()
    assert plan[0] and stat["converged"] == 1
    return got, plan[1]


def _volumes(rng, shape):
    raw = (rng.random(shape) < 0.5).astype(np.uint8)
    return [blobs3d(rng, *shape, max(2, np.prod(shape) // 2000), rmax=9), raw, np.ones(shape, np.uint8)]


# the third and fourth shapes can be cut along one axis only
@pytest.mark.parametrize("slab_voxels", [10000, 25000])
@pytest.mark.parametrize("shape", [(64, 128, 30), (40, 60, 24), (7, 250, 29), (250, 8, 30), (300, 200, 1), (100, 110, 9),
                                   (40, 41, 31), (30, 44, 65)])
def test_boxes(ctx, shape, slab_voxels, monkeypatch):
    monkeypatch.setenv("BGT_RES3D_SLAB_VOXELS", str(slab_voxels))
    for v in _volumes(np.random.default_rng(sum(shape)), shape):
        got, boxes = _thin(ctx, v)
        want = po.thin3d(v)[0]
        assert boxes > 1
        assert np.array_equal(got, want), f"{boxes} boxes: {(got != want).sum()} voxels differ"


@pytest.mark.parametrize("shape", [(200, 200, 24), (64, 128, 30), (96, 96, 16), (8192, 1, 30)])
def test_planned_boxes(ctx, shape):
    """As the planner cuts them by itself."""
    for v in _volumes(np.random.default_rng(sum(shape)), shape):
        got, boxes = _thin(ctx, v)
        want = po.thin3d(v)[0]
        assert boxes > 1
        assert np.array_equal(got, want), f"{boxes} boxes: {(got != want).sum()} voxels differ"


@pytest.mark.parametrize("fill", [0.6, 1.0])
@pytest.mark.parametrize("shape", [(100, 110, 30), (100, 110, 7), (64, 100, 31)])
def test_more_words_than_the_lists_hold(ctx, shape, fill):
    rng = np.random.default_rng(7)
    v = (rng.random(shape) < fill).astype(np.uint8)
    got, boxes = _thin(ctx, v, grid=1)
    want = po.thin3d(v)[0]
    assert boxes == 1
    assert np.array_equal(got, want), f"{(got != want).sum()} voxels differ"
