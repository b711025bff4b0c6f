"""GPU parity of volumes with more non-empty words than a box's lists hold
(begputhinning_b200/csrc/resident.cu: box_collect_all): solids, whose
candidates of an iteration are listed all the same, masks with more candidates
than fit the lists in their first iterations and fewer later on, in one box
and in several."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _solid(kind, shape):
    rng = np.random.default_rng(sum(shape))
    z, y, x = np.mgrid[0:shape[0], 0:shape[1], 0:shape[2]]
    if kind == "full":
        return np.ones(shape, np.uint8)
    if kind == "ball":
        c = [(n - 1) / 2 for n in shape]
        return (sum(((k - m) / (m + 0.1)) ** 2 for k, m in zip((z, y, x), c)) <= 1).astype(np.uint8)
    if kind == "holes":
        return (rng.random(shape) > 0.004).astype(np.uint8)
    if kind == "noise":
        return (rng.random(shape) < 0.6).astype(np.uint8)
    a = (rng.random(shape) < 0.5).astype(np.uint8)  # half noise, half solid
    a[:, shape[1] // 2:] = 1
    return a


@pytest.mark.parametrize("kind", ["full", "ball", "holes", "noise", "half"])
@pytest.mark.parametrize("shape,grid", [((64, 64, 64), 1), ((60, 130, 31), 1), ((100, 110, 30), 1), ((40, 40, 200), 1),
                                        ((70, 130, 126), 12), ((30, 60, 400), 4)])
def test_solids(ctx, shape, grid, kind):
    import torch
    from begputhinning_b200 import Batch, BGTError
    v = _solid(kind, shape)
    want, iterations = po.thin3d(v)
    b = Batch(ctx)
    try:
        i = b.add(shape)
        b.set_grid(grid)
        b.finalize()
        t = torch.from_numpy(v).cuda()
        o = torch.full_like(t, 7)
        b.set_io(i, t, o)
        b.run()
        assert b.plan(i)[0]
        if iterations > max(shape) + 27:  # past the engine's cap of passes: said so, not half done
            with pytest.raises(BGTError, match="pass cap"):
                b.stats(i)
            return
        got, stat = o.cpu().numpy(), b.stats(i)
    finally:
        b.close()
    assert stat["converged"] == 1
    assert np.array_equal(got, want), f"{(got != want).sum()} voxels differ"
