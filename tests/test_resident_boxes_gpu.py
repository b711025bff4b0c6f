"""GPU parity of the resident kernel's boxes (begputhinning_b200/csrc/resident.cu)
against the oracle: one box, cuts along y, along z and along both, boxes whose
cores are as thin as the halo, ragged and word-boundary widths, change masks
with more than one word per column, and boxes with more non-empty words than
their lists hold; images cut along rows, along words and along both."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.helpers import blobs2d, blobs3d, random2d, random3d

pytestmark = pytest.mark.gpu


def _thin(ctx, vols, grid=0):
    import torch
    from begputhinning_b200 import Batch
    b = Batch(ctx)
    ids = [b.add(v.shape) for v in vols]
    if grid:
        b.set_grid(grid)
    b.finalize()
    ins = [torch.from_numpy(v).cuda() for v in vols]
    outs = [torch.full_like(t, 7) for t in ins]
    for i, t, o in zip(ids, ins, outs):
        b.set_io(i, t, o)
    for _ in range(2):
        b.run()
    res = [o.cpu().numpy() for o in outs], [b.plan(i) for i in ids], [b.stats(i) for i in ids]
    b.close()
    return res


@pytest.mark.parametrize("box_words", [20, 200, 3000, 1000000])
@pytest.mark.parametrize("shape", [(13, 14, 31), (12, 70, 32), (70, 12, 33), (40, 41, 65), (7, 90, 97), (25, 24, 1100)])
def test_boxes(ctx, shape, box_words, monkeypatch):
    monkeypatch.setenv("BGT_RES3D_BOX_WORDS", str(box_words))
    rng = np.random.default_rng(sum(shape))
    vols = [random3d(rng, *shape, 0.5), blobs3d(rng, *shape, max(2, np.prod(shape) // 2000), rmax=9),
            np.ones(shape, np.uint8)]
    for v in vols:  # one volume per batch: its share of the work is the whole grid
        (got,), (plan,), (stat,) = _thin(ctx, [v])
        want, _ = po.thin3d(v)
        assert plan[0] and stat["converged"] == 1
        assert np.array_equal(got, want), f"plan {plan}: {(got != want).sum()} voxels differ"


@pytest.mark.parametrize("density", [0.02, 0.6])
def test_boxes_dense(ctx, density):
    """Few CTAs, so large boxes: the sparse volume's words fit the lists, the
    dense one's do not and every word is gone over."""
    rng = np.random.default_rng(3)
    vols = [random3d(rng, 70, 130, 126, density), blobs3d(rng, 30, 30, 40, 5)]
    got, plans, stats = _thin(ctx, vols, grid=12)
    assert all(p[0] for p in plans)
    for g, v, s in zip(got, vols, stats):
        assert s["converged"] == 1
        assert np.array_equal(g, po.thin3d(v)[0]), f"{plans}"


@pytest.mark.parametrize("box_words", [30, 200, 1000000])
@pytest.mark.parametrize("shape", [(24, 300), (75, 260), (200, 129), (333, 1001), (97, 4000), (1500, 40)])
def test_image_boxes(ctx, shape, box_words, monkeypatch):
    monkeypatch.setenv("BGT_RES2D_BOX_WORDS", str(box_words))
    rng = np.random.default_rng(sum(shape))
    for v in (random2d(rng, *shape, 0.5), blobs2d(rng, *shape, max(2, np.prod(shape) // 3000), rmax=14),
              np.ones(shape, np.uint8)):
        (got,), (plan,), (stat,) = _thin(ctx, [v])
        want, _ = po.thin2d(v)
        assert plan[0] and stat["converged"] == 1
        assert np.array_equal(got, want), f"plan {plan}: {(got != want).sum()} pixels differ"


def wedges2d(h, w):
    """Wide wedges in all four directions: deletions travel along them for many
    passes, so words fall out of a pass, come back, and pass on to their
    neighbours at different times."""
    y, x = np.mgrid[0:h, 0:w]
    v = (np.abs(y - h // 2) * 3 < x % 150) | (np.abs(x - w // 2) * 3 < (h - y) % 130)
    v[:, ::97] = 0
    return v.astype(np.uint8)


# units of 2, 4 and 8 words; unit rows and words cut anywhere
@pytest.mark.parametrize("shape", [(60, 70), (97, 159), (230, 257), (310, 700), (767, 1025)])
def test_active_words(ctx, shape):
    for v in (wedges2d(*shape), wedges2d(shape[0], shape[1] + 5)[::-1, 5:].copy()):
        (got,), _, (stat,) = _thin(ctx, [v])
        assert stat["converged"] == 1
        assert np.array_equal(got, po.thin2d(v)[0]), f"{(got != po.thin2d(v)[0]).sum()} pixels differ"


@pytest.mark.parametrize("slab_voxels", [10000, 40000])
def test_messages_of_earlier_runs(ctx, slab_voxels, monkeypatch):
    """A batch run again and again on other volumes, and batches made anew in the
    memory that the last one left: the boxes take over this run's messages only."""
    import torch
    from begputhinning_b200 import Batch
    monkeypatch.setenv("BGT_RES3D_SLAB_VOXELS", str(slab_voxels))
    rng = np.random.default_rng(60)
    shape = (31, 44, 70)
    vols = [blobs3d(rng, *shape, 9, rmax=8), np.ones(shape, np.uint8), random3d(rng, *shape, 0.6),
            blobs3d(rng, *shape, 30, rmax=5)]
    wants = [po.thin3d(v)[0] for v in vols]
    t = torch.empty(shape, dtype=torch.uint8, device="cuda")
    o = torch.empty_like(t)
    for k in range(3):
        b = Batch(ctx)
        i = b.add(shape)
        b.finalize()
        b.set_io(i, t, o)
        assert b.plan(i)[1] > 1
        for v, want in list(zip(vols, wants))[::-1 if k == 1 else 1]:
            t.copy_(torch.from_numpy(v))
            torch.cuda.synchronize()
            b.run()
            torch.cuda.synchronize()
            assert np.array_equal(o.cpu().numpy(), want)
        b.close()
