"""Workloads of the library as its users run them, for timing.

``listed()`` names the workloads, ``draw(rng)`` gives another one of the same
ranges, ``prepare`` makes the inputs and whatever a program keeps between
calls (a batch, an output buffer), ``run`` makes one pass through the public
API, ``work`` says what a pass cannot do without, and ``exact`` restates the
floating-point outputs in 64 bits with numpy alone.

Kinds of case:

* ``thin2d`` / ``thin3d``: ``thin_device`` on one image or volume in device memory
* ``batch``: ``Batch.run`` on many images and volumes of uneven size
* ``segments2d`` / ``segments3d``: ``ExtractSegmentsV`` on a thinned mask in device memory
* ``centerline2d`` / ``centerline3d``: ``CenterlineExtraction`` on a host array,
  the reference's whole path (thinning, segments, pruning, smoothing)
"""
from __future__ import annotations

import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import begputhinning_b200 as bgt
from begputhinning_b200 import synth

ITEM_BYTES = {"uint8": 1, "int16": 2, "float32": 4}


def listed():
    return [
        # a small crop, one call: launches and host work are the time
        {"name": "crop_200x160", "kind": "thin2d", "w": 200, "h": 160, "content": "strokes", "dtype": "uint8"},
        # the plain 2D image: 12 strokes in 512 x 512
        {"name": "frame_512", "kind": "thin2d", "w": 512, "h": 512, "content": "strokes", "dtype": "uint8"},
        # a float mask of odd size, as a segmentation network hands it over
        {"name": "image_f32_1501x1003", "kind": "thin2d", "w": 1501, "h": 1003, "content": "strokes",
         "dtype": "float32"},
        # the large 2D image: vessel trees with salt and holes
        {"name": "vessels_4096", "kind": "thin2d", "w": 4096, "h": 4096, "content": "vessels", "dtype": "uint8"},
        # a small volume of ragged size: a region of interest
        {"name": "roi_97x75x66", "kind": "thin3d", "w": 97, "h": 75, "d": 66, "dtype": "uint8"},
        # the plain 3D volume: trees and solid ellipsoids in 256^3
        {"name": "trees_256", "kind": "thin3d", "w": 256, "h": 256, "d": 256, "dtype": "uint8"},
        # one frame of each of 16 camera streams, thinned together
        {"name": "frames_16x1024", "kind": "batch", "n2d": 16, "n3d": 0, "side": 1024, "shapes": 4,
         "dtype": "uint8"},
        # the batched workload: 512 images and 32 volumes of uneven size
        {"name": "mixed_512_32", "kind": "batch", "n2d": 512, "n3d": 32, "side": 0, "shapes": 3, "dtype": "uint8"},
        # segments of a large thinned image that stayed on the device
        {"name": "segments_2048", "kind": "segments2d", "w": 2048, "h": 2048, "content": "strokes",
         "dtype": "uint8"},
        # segments of the thinned 256^3 volume
        {"name": "segments_256x3", "kind": "segments3d", "w": 256, "h": 256, "d": 256, "dtype": "uint8"},
        # the whole path on the plain 2D image, from host memory to host memory
        {"name": "centerline_512", "kind": "centerline2d", "w": 512, "h": 512, "content": "strokes",
         "dtype": "uint8", "prune": 5, "span": 3},
        # the whole path on a 16-bit volume of odd size
        {"name": "centerline_i16_187x203x161", "kind": "centerline3d", "w": 187, "h": 203, "d": 161,
         "dtype": "int16", "prune": 4, "span": 2},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _image_size(rng, lo, hi):
    w = _log_uniform(rng, lo, hi)
    return w, min(hi, max(lo, int(round(w * math.exp(rng.uniform(math.log(0.5), math.log(2.0)))))))


def draw(rng):
    kind = rng.choice(["thin2d", "thin2d", "thin3d", "thin3d", "batch", "batch", "segments2d", "segments3d",
                       "centerline2d", "centerline3d"])
    if kind == "batch":
        side = rng.choice([0, 0, _log_uniform(rng, 200, 1024)])
        n2d = _log_uniform(rng, 4, min(512, (1 << 27) // side ** 2) if side else 512)
        return {"kind": kind, "n2d": n2d, "n3d": rng.choice([0, _log_uniform(rng, 1, 32)]), "side": side,
                "shapes": rng.randrange(1 << 20), "dtype": "uint8"}
    case = {"kind": kind, "dtype": rng.choice(["uint8", "uint8", "int16", "float32"])}
    if kind.endswith("3d"):
        hi = 203 if kind == "centerline3d" else 256
        case.update(w=_log_uniform(rng, 64, hi), h=_log_uniform(rng, 64, hi), d=_log_uniform(rng, 64, hi))
    else:
        lo, hi = {"thin2d": (64, 4096), "segments2d": (128, 2048), "centerline2d": (64, 1024)}[kind]
        case["w"], case["h"] = _image_size(rng, lo, hi)
        case["content"] = rng.choice(["strokes", "vessels"]) if min(case["w"], case["h"]) >= 512 else "strokes"
    if kind.startswith("centerline"):
        case.update(prune=rng.randrange(0, 12), span=rng.randrange(0, 6))
    return case


# ------------------------------------------------------------- inputs -----
def _image(seed, w, h, content="strokes"):
    """Seeded uint8 {0,1} image: strokes at 12 per 512^2, or vessel trees at 20 per 4096^2."""
    area = w * h
    if content == "vessels":
        return synth.vessels2d(seed, w, h, nroots=max(1, round(20 * area / 4096 ** 2)),
                               nholes=round(50 * area / 4096 ** 2))
    return synth.strokes2d(seed, w, h, max(1, round(12 * area / 512 ** 2)))


def _volume(seed, w, h, d):
    """Seeded uint8 {0,1} volume: 8 trees and 3 ellipsoids per 256^3."""
    share = w * h * d / 256 ** 3
    return synth.trees3d(seed, w, h, d, ntrees=max(1, round(8 * share)), nell=round(3 * share))


def _host_input(case, seed):
    if case["kind"].endswith("3d"):
        a = _volume(seed, case["w"], case["h"], case["d"])
    else:
        a = _image(seed, case["w"], case["h"], case["content"])
    return a.astype(case["dtype"])


def _batch_shapes(case):
    """(h, w) and (d, h, w) of the instances: fixed by the case, not by the seed."""
    if case["side"]:
        twod = [(case["side"], case["side"])] * case["n2d"]
        threed = [(d, h, w) for w, h, d, _, _ in synth.mixed_batch_shapes(case["shapes"], 0, case["n3d"])[1]]
    else:
        s2, s3 = synth.mixed_batch_shapes(case["shapes"], case["n2d"], case["n3d"])
        twod = [(h, w) for w, h, _ in s2]
        threed = [(d, h, w) for w, h, d, _, _ in s3]
    return twod + threed


def _batch_state(case, seed):
    shapes = _batch_shapes(case)
    sizes = [math.prod(s) for s in shapes]
    offs = np.cumsum([0] + sizes)
    host = np.empty(int(offs[-1]), np.uint8)

    def fill(i):
        s = shapes[i]
        a = _image(seed * 1000003 + i, s[1], s[0]) if len(s) == 2 else _volume(seed * 1000003 + i, s[2], s[1], s[0])
        host[offs[i]:offs[i + 1]] = a.reshape(-1)

    with ThreadPoolExecutor(8) as pool:
        list(pool.map(fill, sorted(range(len(shapes)), key=lambda i: -sizes[i])))
    dev_in = torch.from_numpy(host).cuda()
    dev_out = torch.zeros_like(dev_in)
    batch = bgt.Batch()
    ids = [batch.add(s) for s in shapes]
    batch.finalize()
    for k, i in enumerate(ids):
        lo, hi = int(offs[k]), int(offs[k + 1])
        batch.set_io(i, dev_in[lo:hi], dev_out[lo:hi])
    return {"batch": batch, "in": dev_in, "out": dev_out}


def _room(case):
    """Points and segments that the program keeps room for: more than any
    image or volume of the case's size and content holds."""
    n = case["w"] * case["h"] * case.get("d", 1)
    return (n // 1024 + 2048, n // 8192 + 512) if case["kind"].endswith("3d") else (n // 12 + 1024, n // 64 + 512)


def _lists(case):
    """Host arrays of a fixed size that the lists are collected in (zeros after their end)."""
    points, segs = _room(case)
    dims = 3 if case["kind"].endswith("3d") else 2
    if case["kind"].startswith("segments"):
        return [np.zeros(segs + 1, np.int32), np.zeros(segs, np.uint8), np.zeros((points, dims), np.int16)]
    return [np.zeros(points, np.float32) for _ in range(dims)] + [np.zeros(segs + 1, np.uint32)]


def _collect(lists, parts):
    for a, p in zip(lists, parts):
        a[:len(p)] = p
        a[len(p):] = 0
    return [*lists, len(parts[0])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"case": case, **_batch_state(case, seed)}
    a = _host_input(case, seed)
    if kind.startswith("centerline"):
        return {"case": case, "in": a, "lists": _lists(case)}
    t = torch.from_numpy(a).cuda()
    if kind.startswith("segments"):
        return {"case": case, "in": bgt.thin_device(t), "lists": _lists(case)}
    return {"case": case, "in": t, "out": torch.zeros_like(t)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].run()
        return state["out"]
    if kind.startswith("thin"):
        return bgt.thin_device(state["in"], state["out"])
    if kind.startswith("segments"):
        s = bgt.ExtractSegmentsV(state["in"])
        return _collect(state["lists"], (s.start, s.is_end, s.pts))
    return _collect(state["lists"], bgt.CenterlineExtraction(state["in"], case["prune"], case["span"]))


def work(case):
    """Bytes of the pixels read once and, for thinned masks, written once
    (segment lists are a small fraction of that); the operations on them are
    bitwise, none is a floating-point one."""
    if case["kind"] == "batch":
        return {"bytes": 2 * sum(math.prod(s) for s in _batch_shapes(case)), "flops": 0}
    n = case["w"] * case["h"] * case.get("d", 1) * ITEM_BYTES[case["dtype"]]
    return {"bytes": 2 * n if case["kind"].startswith("thin") else n, "flops": 0}


# -------------------------------------------- 64-bit restatement (numpy) --
def _thin2d_exact(fg):
    """N, S, E, W subiterations until one whole iteration deletes nothing
    (2D/CUDA_SubiterationKernels2D.cuh:15-119)."""
    h, w = fg.shape
    p = np.zeros((h + 2, w + 2), bool)
    p[1:-1, 1:-1] = fg
    ring = [(-1, 0), (-1, 1), (0, 1), (1, 1), (1, 0), (1, -1), (0, -1), (-1, -1)]
    while True:
        before = int(p.sum())
        for r in (0, 4, 2, 6):
            # only rows and columns that hold foreground are looked at
            ys, xs = np.nonzero(p)
            x = [p[ys + ring[(k + r) & 7][0], xs + ring[(k + r) & 7][1]] for k in range(8)]
            a = ~x[1] & ~x[7] & (x[2] ^ x[3] ^ ~x[4]) & (x[3] ^ x[5]) & (x[3] ^ x[6])
            b = x[2] & x[4] & (x[6] | ~x[7])
            c = ~x[1] & x[4] & x[6]
            d = ~x[6] & ~x[7] & (x[1] ^ x[5]) & (x[2] ^ x[5]) & (x[4] ^ ~x[5])
            e = ~x[1] & ~x[2] & ~x[3] & x[6] & x[7]
            gone = ~x[0] & (a | b | c | d | e)
            p[ys[gone], xs[gone]] = False
        if int(p.sum()) == before:
            return p[1:-1, 1:-1].copy()


def _rule3d_exact(n, perm, sign):
    """Deletable flags of one direction (3D/CUDA_SubiterationKernels3D.cuh:14-234):
    the "up" rule in the frame that the axis order and sign of the direction give."""
    def g(a, b, c):
        off = [0, 0, 0]
        for k, v in zip(perm, (sign * a, b, c)):
            off[k] = v
        return n[9 * (off[0] + 1) + 3 * (off[1] + 1) + off[2] + 1]

    tn, ts, tw, te = g(-1, -1, 0), g(-1, 1, 0), g(-1, 0, -1), g(-1, 0, 1)
    tnw, tne, tsw, tse = g(-1, -1, -1), g(-1, -1, 1), g(-1, 1, -1), g(-1, 1, 1)
    mn, ms, mw, me = g(0, -1, 0), g(0, 1, 0), g(0, 0, -1), g(0, 0, 1)
    mnw, mne, msw, mse = g(0, -1, -1), g(0, -1, 1), g(0, 1, -1), g(0, 1, 1)
    bn, bs, bw, be = g(1, -1, 0), g(1, 1, 0), g(1, 0, -1), g(1, 0, 1)
    bnw, bne, bsw, bse = g(1, -1, -1), g(1, -1, 1), g(1, 1, -1), g(1, 1, 1)
    t, b = g(-1, 0, 0), g(1, 0, 0)
    mid = mnw | mn | mne | mw | me | msw | ms | mse | bnw | bne | bsw | bse
    arm_n, arm_s = bn & ~bs & ~ms & ~mse & ~bse, bs & ~bn & ~mn & ~mne & ~bne
    arm_w, arm_e = bw & ~be & ~me, be & ~bw & ~mw
    east_s, east_n = arm_e & ~msw & ~bsw, arm_e & ~mnw & ~bnw
    m1 = mid | bw | be | bn | bs
    m5 = ((mid | bw | be) & ((arm_n & ~msw & ~bsw) | (arm_s & ~mnw & ~bnw))) | (
        (mid | bn | bs) & ((east_n & ~msw & ~bsw) | (arm_w & ~mne & ~mse & ~bne & ~bse)))
    m6 = (east_s & bn & ~bs & ~ms) | (east_n & bs & ~bn & ~mn) | (arm_w & (arm_n | arm_s))
    m4 = (~tnw & ~tsw & ((tne & mne & ~tse) | (tse & mse & ~tne))) | (
        ~tne & ~tse & ((tnw & mnw & ~tsw) | (tsw & msw & ~tnw)))
    m2 = (~tn & ~tne & ~te & ((~tnw & ~tw & ms) | (~ts & ~tse & mw))) | (
        ~ts & ~tsw & ~tw & ((~te & ~tse & mn) | (~tnw & ~tn & me)))
    m3 = (~tw & me & ((~ts & ~tsw & mn) | (~tnw & ~tn & ms))) | (~te & mw & ((~tn & ~tne & ms) | (~ts & ~tse & mn)))
    cross, corner = ~(tn | tw | te | ts), ~(tnw | tne | tsw | tse)
    return ~t & ((cross & ((b & m4) | (corner & ((b & m1) | (~b & (m5 | m6)))))) | (b & (m2 | m3)))


def _thin3d_exact(fg):
    """Pre-test, then U, N, E, D, S, W on its union, until an iteration
    deletes nothing (3D/CUDA_ThinningKernel3D_Linear.cuh:746-782)."""
    d, h, w = fg.shape
    p = np.zeros((d + 2, h + 2, w + 2), bool)
    p[1:-1, 1:-1, 1:-1] = fg
    flat = p.reshape(-1)
    row, plane = w + 2, (w + 2) * (h + 2)
    offs = [dz * plane + dy * row + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    dirs = [((0, 1, 2), 1), ((1, 0, 2), 1), ((2, 0, 1), 1), ((0, 1, 2), -1), ((1, 0, 2), -1), ((2, 0, 1), -1)]
    pts = np.flatnonzero(flat)
    while True:
        n = [flat[pts + o] for o in offs]
        union = np.zeros(len(pts), bool)
        for d6 in dirs:
            union |= _rule3d_exact(n, *d6)
        todo = pts[union]
        for d6 in dirs:
            todo = todo[flat[todo]]
            gone = _rule3d_exact([flat[todo + o] for o in offs], *d6)
            flat[todo[gone]] = False
        left = pts[flat[pts]]
        if len(left) == len(pts):
            return p[1:-1, 1:-1, 1:-1].copy()
        pts = left


def _segments_exact(fg):
    """The raster-order walk (2D/ExtractSegments.cpp:16-127,
    3D/ExtractSegments.cpp:135-251): [(is_end, [linear index, ...]), ...]."""
    shape = fg.shape
    strides = [math.prod(shape[k + 1:]) for k in range(fg.ndim)]
    steps = [()]
    for _ in shape:
        steps = [s + (k,) for s in steps for k in (-1, 0, 1)]
    delta = [sum(a * b for a, b in zip(s, strides)) for s in steps if any(s)]
    inner = np.zeros(shape, bool)
    inner[(slice(1, -1),) * fg.ndim] = fg[(slice(1, -1),) * fg.ndim]
    flat = fg.reshape(-1)
    pts = np.flatnonzero(inner)
    count = sum((flat[pts + o].astype(int) for o in delta), np.zeros(len(pts), int))
    first = {int(i): (2 if c == 2 else -max(int(c), 1)) for i, c in zip(pts, count)}
    val = dict(first)
    segs = []
    for p in map(int, pts):
        budget = val[p]
        if budget >= 0:
            continue
        val[p] = 0
        nxt = 0
        for _ in range(-budget):
            end, path = abs(first[p]) < 2, [p]
            while nxt < len(delta) and not val.get(p + delta[nxt], 0):
                nxt += 1
            if nxt < len(delta):
                t = p + delta[nxt]
                nxt += 1
                while val[t] == 2:
                    val[t] = 0
                    path.append(t)
                    t = next((t + o for o in delta if val.get(t + o, 0)), t)
                path.append(t)
                end = end or abs(first[t]) < 2
                val[t] += 1
            else:
                nxt += 1
            segs.append((end, path))
    return segs


def _centerline_exact(case, seed):
    a = _host_input(case, seed) > 0
    pad = [((n + 31) // 32) * 32 for n in a.shape]
    if a.ndim == 2:
        pad[0] = max(1, (a.shape[0] + 63) // 128) * 128 + 64
    full = np.zeros(pad, bool)
    full[tuple(slice(0, min(n, m)) for n, m in zip(a.shape, pad))] = a
    thin = (_thin2d_exact if a.ndim == 2 else _thin3d_exact)(full)
    cols = [[] for _ in pad]
    for end, path in _segments_exact(thin):
        n = len(path)
        if end and n <= case["prune"]:
            continue
        span = min(case["span"], (n - 1) // 2)
        q = np.arange(n)
        half = np.minimum(span, np.minimum(q, n - 1 - q))
        for k, c in enumerate(np.unravel_index(np.array(path), pad)):
            total = np.concatenate([[0], np.cumsum(c.astype(np.int64))])
            cols[k].append((total[q + half + 1] - total[q - half]) / (2.0 * half + 1.0))
    room = _room(case)[0]
    out = [np.concatenate(c) if c else np.zeros(0) for c in reversed(cols)]
    return [*(np.concatenate([c, np.zeros(room - len(c))]) for c in out), None, None]


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("centerline"):
        return _centerline_exact(case, seed)
    if kind == "thin2d" and case["dtype"] == "float32":
        return torch.from_numpy(_thin2d_exact(_host_input(case, seed) >= 1).astype(np.float64))
    if kind == "thin3d" and case["dtype"] == "float32":
        return torch.from_numpy(_thin3d_exact(_host_input(case, seed) >= 1).astype(np.float64))
    return None  # masks and segment lists are whole numbers
