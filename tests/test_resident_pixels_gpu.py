"""GPU parity of the resident kernel's own pixel reads and writes
(begputhinning_b200/csrc/pixels.cuh) against the oracle: every pixel type and
its foreground rule, arrays that start at any element of a larger one (the
bytes around the output stay as they were), widths at the edges of words and
chunks, outputs over inputs, and an output that is another instance's input."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

DTYPES = ["uint8", "int8", "bool", "uint16", "int16", "uint32", "int32", "float32", "float64"]


def _values(rng, shape, dtype):
    """Blobs of values whose foreground test differs between the types and the dimensions."""
    v = rng.integers(-3, 6, shape)
    v[rng.random(shape) < 0.35] = 0
    if dtype == "bool":
        return v > 0
    if dtype.startswith("f"):
        return (v * 0.5).astype(dtype)
    info = np.iinfo(dtype)
    return (v & info.max if info.min == 0 else v).astype(dtype)


def _want(a):
    from begputhinning_b200.api import dtype_code
    fg = po.binarise(np.ascontiguousarray(a), dtype_code(a.dtype), a.ndim).reshape(a.shape)
    return (po.thin2d if a.ndim == 2 else po.thin3d)(fg)[0]


def _placed(a, skip):
    """The array inside a larger CUDA tensor, `skip` elements after its start."""
    import torch
    n = a.size
    big = torch.from_numpy(np.full(n + 128, 9).astype(a.dtype)).cuda()
    view = big[skip:skip + n].view(a.shape)
    view.copy_(torch.from_numpy(a))
    return big, view


def _run(ctx, views):
    from begputhinning_b200 import Batch
    b = Batch(ctx)
    ids = [b.add(tuple(i.shape)) for i, _ in views]
    b.finalize()
    for k, (i, o) in zip(ids, views):
        b.set_io(k, i, o)
    b.run()
    assert all(b.plan(k)[0] for k in ids)
    b.close()


@pytest.mark.parametrize("shape", [(70, 1), (40, 31), (33, 33), (37, 47), (64, 64), (90, 100), (300, 129), (9, 20, 33),
                                   (20, 31, 64), (40, 40, 70)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_types_and_offsets(ctx, dtype, shape):
    rng = np.random.default_rng(sum(shape) + DTYPES.index(dtype))
    views, checks = [], []
    for skip_in, skip_out in ((0, 0), (1, 3), (13, 31), (17, 16)):
        a = _values(rng, shape, dtype)
        _, i = _placed(a, skip_in)
        big, o = _placed(a, skip_out)
        views.append((i, o))
        checks.append((a, big, o, skip_out))
    _run(ctx, views)
    for a, big, o, skip in checks:
        assert np.array_equal(o.cpu().numpy(), _want(a).astype(a.dtype))
        rest = big.cpu().numpy()
        assert (rest[:skip] == np.array(9).astype(a.dtype)).all() and (rest[skip + a.size:] == np.array(9).astype(a.dtype)).all()


@pytest.mark.parametrize("dims", [2, 3])
def test_shared_arrays(ctx, dims):
    import torch
    rng = np.random.default_rng(dims)
    shape = (300, 200) if dims == 2 else (30, 40, 50)
    a, c = ((rng.random(shape) < 0.6).astype(np.uint8) for _ in range(2))
    t, u = torch.from_numpy(a).cuda(), torch.from_numpy(c).cuda()
    v = torch.zeros_like(t)
    _run(ctx, [(t, t)])  # in place
    assert np.array_equal(t.cpu().numpy(), _want(a))
    t.copy_(torch.from_numpy(a))
    _run(ctx, [(t, u), (u, v)])  # the second's input is overwritten by the first's output: all inputs are read first
    assert np.array_equal(u.cpu().numpy(), _want(a)) and np.array_equal(v.cpu().numpy(), _want(c))


@pytest.mark.parametrize("dims", [2, 3])
def test_padded_shape_then_plain(ctx, dims):
    """The shape that CenterlineExtraction pads an input to, thinned afterwards
    through the same context: the whole array is read."""
    import torch
    from begputhinning_b200 import CenterlineExtraction, Thinning2D, Thinning3D, thin_device
    rng = np.random.default_rng(dims)
    small, full = ((100, 20), (192, 32)) if dims == 2 else ((20, 25, 30), (32, 32, 32))
    a = (rng.random(full) < 0.6).astype(np.uint8)
    CenterlineExtraction((rng.random(small) < 0.6).astype(np.uint8), 2, 1, ctx)
    assert np.array_equal(thin_device(torch.from_numpy(a).cuda(), ctx=ctx).cpu().numpy(), _want(a))
    CenterlineExtraction((rng.random(small) < 0.6).astype(np.uint8), 2, 1, ctx)
    assert np.array_equal((Thinning2D if dims == 2 else Thinning3D)(a, ctx), _want(a))
