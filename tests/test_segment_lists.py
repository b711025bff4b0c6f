"""CenterlineExtraction of skeletons with more segments per node than the
lists are sized for at first (begputhinning_b200/csrc/segments_graph.cu):
checkerboards, whose voxels are not simple and have twelve neighbours each, so
that a node has up to six segments of two points.  Their segments fit the
output block, which is sized for longer ones, but not the list of the kept
segments: the extraction has to be run again with a longer list."""
import numpy as np
import pytest

from oracle import pyoracle as po


def _checkerboard(n):
    z, y, x = np.mgrid[0:n, 0:n, 0:n]
    return np.pad(((x + y + z) % 2 == 0).astype(np.uint8), 2)


@pytest.mark.parametrize("n,more", [(18, False), (19, True), (20, True)])
def test_checkerboards_are_such_skeletons(n, more):
    t = po.thin3d(_checkerboard(n))[0]
    s = po.segments3d(t)
    # lists of a 32^3 volume: 4096 nodes, 16384 chain points; four segments and eight points per node
    nodes, segs, points = 4096, 4 * 4096, 16384 + 8 * 4096
    assert int(t.sum()) <= nodes
    assert 5 * s.nseg + 6 * len(s.pts) <= 5 * segs + 6 * points
    assert (s.nseg > segs) == more


@pytest.mark.gpu
@pytest.mark.parametrize("n", [18, 19, 20])
@pytest.mark.parametrize("prune,span", [(0, 1), (3, 2), (-1, 0)])
def test_centerlines_of_checkerboards(ctx, n, prune, span):
    from begputhinning_b200 import CenterlineExtraction, Context
    v = _checkerboard(n)
    want = po.centerline3d(v, prune, span)
    c = Context(0)  # whose lists have not grown yet
    for _ in range(2):
        got = CenterlineExtraction(v, prune, span, c)
        for g, w in zip(got, (want.x, want.y, want.z, want.idx), strict=True):
            assert np.array_equal(g, w)
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["segments", "centerline"])
def test_results_of_more_than_256_mb(ctx, kind):
    """They come back through memory that the context does not keep."""
    from begputhinning_b200 import CenterlineExtraction, ExtractSegmentsV
    if kind == "segments":
        a = (np.random.default_rng(4).random((4700, 5000)) < 0.5).astype(np.uint8)
        want = po.segments2d(a)
        assert 5 * want.nseg + 4 * len(want.pts) > 256 << 20
        got = ExtractSegmentsV(a, ctx)
        for g, w in ((got.start, want.start), (got.is_end, want.is_end), (got.pts, want.pts)):
            assert np.array_equal(g, w)
    else:
        v = _checkerboard(150)
        want = po.centerline3d(v, 1, 1)
        assert 12 * len(want.x) + 4 * len(want.idx) > 256 << 20
        for g, w in zip(CenterlineExtraction(v, 1, 1, ctx), (want.x, want.y, want.z, want.idx), strict=True):
            assert np.array_equal(g, w)
    small = (np.random.default_rng(5).random((60, 70)) < 0.3).astype(np.uint8)
    assert ExtractSegmentsV(small, ctx).as_lists() == po.segments2d(small).as_lists()
