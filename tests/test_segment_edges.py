"""The closed form of the reference's segment walk that the one-launch
extraction (begputhinning_b200/csrc/segments_graph.cu) implements: every edge
of the skeleton graph is walked by its raster-earlier node, so each node's
segments follow from its own neighbours alone.  CPU: a plain restatement of
that form against the oracle, on thinned and raw masks, frame pixels
included.  GPU: the kernel against the oracle where its lists, prefix sums
and pointer jumping have their edges (word boundaries, long chains, cycles
without a node, chains back to their own node, lists that must grow)."""
import numpy as np
import pytest

from oracle import pyoracle as po


def edge_model(fg):
    dims = fg.ndim
    steps = [()]
    for _ in fg.shape:
        steps = [s + (k,) for s in steps for k in (-1, 0, 1)]
    steps = [s for s in steps if any(s)]
    last = len(steps) - 1
    inner = np.zeros(fg.shape, bool)
    inner[(slice(1, -1),) * dims] = fg[(slice(1, -1),) * dims] > 0
    points = [tuple(map(int, p)) for p in np.argwhere(inner)]

    def add(p, d):
        return tuple(a + b for a, b in zip(p, steps[d]))

    nbr = {p: [d for d in range(len(steps)) if fg[add(p, d)]] for p in points}
    nodes = {p for p in points if len(nbr[p]) != 2}

    def follow(c, side):
        """Chain points from c on, leaving it on `side`, and the node (and last step) they lead to."""
        path = [c]
        while True:
            d = nbr[c][side]
            n = add(c, d)
            if n not in nbr:
                return path, None, None
            if n in nodes:
                return path, n, d
            c, side = n, int(nbr[n][0] == last - d)
            path.append(c)

    out = []
    for r in points:
        if r not in nodes:
            continue
        n, taken, made = len(nbr[r]), 0, 0
        for d in nbr[r]:
            q = add(r, d)
            if q not in nbr:
                continue
            if q in nodes:
                if q < r:
                    taken += 1
                    continue
                seg = (n < 2 or len(nbr[q]) < 2, [r, q])
            else:
                path, e, de = follow(q, int(nbr[q][0] == last - d))
                if e is None or (e == r and d < last - de):
                    seg = (n < 2, [r, *path, path[-1]])
                elif e == r:
                    seg = (n < 2, [r, q])
                elif e < r:
                    taken += 1
                    continue
                else:
                    seg = (n < 2 or len(nbr[e]) < 2, [r, *path, e])
            out.append(seg)
            made += 1
        out += [(n < 2, [r])] * (max(n, 1) - taken - made)
    return [(int(e), tuple(tuple(reversed(p)) for p in path)) for e, path in out]


@pytest.mark.parametrize("dims,thin", [(2, False), (2, True), (3, False), (3, True)])
def test_closed_form(dims, thin):
    rng = np.random.default_rng(10 * dims + thin)
    for _ in range(60):
        shape = tuple(rng.integers(1, 26 if dims == 2 else 9, dims))
        a = (rng.random(shape) < rng.choice([0.1, 0.25, 0.4, 0.6])).astype(np.uint8)
        if thin:
            a = (po.thin2d if dims == 2 else po.thin3d)(a)[0]
        want = (po.segments2d if dims == 2 else po.segments3d)(a).as_lists()
        assert [(int(e), tuple(map(tuple, p))) for e, p in want] == edge_model(a)


def _serpentine(n):
    """Rows four apart joined by diagonal turns: one chain of about n * n / 4 points."""
    a = np.zeros((n, n), np.uint8)
    lo, hi = 5, n - 6
    for k, y in enumerate(range(2, n - 6, 4)):
        a[y, lo:hi + 1] = 1
        x, d = (hi, 1) if k % 2 == 0 else (lo, -1)
        if y + 4 < n - 6:
            a[y + 1, x + d] = a[y + 2, x + 2 * d] = a[y + 3, x + d] = 1
    return a


def _mask(kind, seed=0):
    rng = np.random.default_rng(seed)
    if kind == "serpentine":
        return _serpentine(203)
    if kind == "rings":  # cycles without a node beside cycles through one
        a = np.zeros((70, 131), np.uint8)
        for k, x in enumerate(range(3, 115, 14)):
            a[10, x:x + 9] = a[18, x:x + 9] = a[10:19, x] = a[10:19, x + 8] = 1
            a[30:39, x] = a[30:39, x + 8] = a[30, x:x + 9] = a[38, x:x + 9] = 1
            a[39:42 + k, x + 4] = 1
        return a
    if kind == "frame":  # lines that run into the frame
        a = np.zeros((65, 97), np.uint8)
        a[20, :] = a[:, 40] = a[50, :30] = a[:7, 70] = 1
        a[60, 5] = a[1, 1] = a[63, 95] = 1
        return a
    if kind == "grow":  # more nodes than the lists hold at first
        return (rng.random((700, 900)) < 0.5).astype(np.uint8)
    if kind == "dense3":
        return (rng.random((20, 33, 65)) < 0.3).astype(np.uint8)
    if kind == "thin3":
        return po.thin3d((rng.random((40, 50, 64)) < 0.35).astype(np.uint8))[0]
    h, w = map(int, kind.split("x"))
    return po.thin2d((rng.random((h, w)) < 0.6).astype(np.uint8))[0]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["serpentine", "rings", "frame", "grow", "dense3", "thin3", "1x1", "2x40", "3x3", "33x31",
                                  "40x32", "64x33", "31x64", "129x65", "500x1030"])
def test_kernel_edges(ctx, kind):
    from begputhinning_b200 import ExtractSegmentsV
    a = _mask(kind)
    want = (po.segments2d if a.ndim == 2 else po.segments3d)(a)
    for _ in range(2):  # the second call finds the lists of the first
        got = ExtractSegmentsV(a, ctx)
        assert got.as_lists() == want.as_lists()


@pytest.mark.gpu
@pytest.mark.parametrize("prune,span", [(0, 0), (3, 1), (12, 7), (-1, 2), (2, -3), (5, 255), (5, 256), (1, 6000)])
@pytest.mark.parametrize("kind", ["serpentine", "frame", "rings", "129x65", "1x1", "thin3"])
def test_centerline_edges(ctx, kind, prune, span):
    """Pruning, smoothing (spans up to and past the one whose running sums stay
    exact) and flattening: the same floats, bit for bit."""
    from begputhinning_b200 import CenterlineExtraction
    a = _mask(kind)
    got = CenterlineExtraction(a, prune, span, ctx)
    want = (po.centerline2d if a.ndim == 2 else po.centerline3d)(a, prune, span)
    arrays = [want.x, want.y] + ([want.z] if a.ndim == 3 else []) + [want.idx]
    for g, w in zip(got, arrays, strict=True):
        assert np.array_equal(g, w)
