"""How a host array reaches the device: packed on the host or byte by byte
(begputhinning_b200/csrc/hostpix.cpp: host_pack_pays).  CPU: the rule at its
edges, and the workers of a process with one CPU.  GPU: the same results on
either side of the rule, from pageable and pinned arrays, on one CPU and on all."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _pays(pixel, nbytes, pinned, workers):
    import ctypes as C
    from begputhinning_b200 import lib
    f = lib()._ZN3bgt14host_pack_paysEmmbi
    f.argtypes, f.restype = [C.c_size_t, C.c_size_t, C.c_bool, C.c_int], C.c_bool
    return f(pixel, nbytes, pinned, workers)


@pytest.mark.parametrize("pixel,nbytes,pinned,workers,pays", [
    (1, 2 << 20, False, 0, True), (1, (2 << 20) + 1, False, 0, False), (2, 12 << 20, False, 0, False),
    (2, 12 << 20, False, 1, True), (4, 64 << 20, False, 0, True), (1, 64, True, 7, False), (4, 1 << 20, True, 2, False),
    (4, 1 << 20, True, 3, True), (8, 1 << 20, True, 7, True)])
def test_rule(pixel, nbytes, pinned, workers, pays):
    assert _pays(pixel, nbytes, pinned, workers) == pays


def _one_cpu(code):
    return subprocess.run([sys.executable, "-c", "import os\nos.sched_setaffinity(0, {min(os.sched_getaffinity(0))})\n" + code],
                          cwd=ROOT, check=True, capture_output=True, text=True).stdout


def test_no_workers_on_one_cpu():
    out = _one_cpu("from begputhinning_b200 import lib\nL = lib()\nL._ZN3bgt16host_pool_retainEv()\n"
                   "print(L._ZN3bgt12host_workersEv())\nL._ZN3bgt17host_pool_releaseEv()")
    assert int(out) == 0


SHAPES = [(100, 70), (1024, 2048), (1025, 2049), (60, 70, 80), (180, 170, 160)]


def _check(ctx, pinned):
    import torch
    from begputhinning_b200 import CenterlineExtraction, Thinning2D, Thinning3D
    from begputhinning_b200 import synth
    from oracle import pyoracle as po
    for shape in SHAPES:
        flat = len(shape) == 2
        a = synth.strokes2d(5, shape[1], shape[0], 40) if flat else synth.trees3d(5, *shape[::-1], ntrees=3, nell=1)
        want = (po.thin2d if flat else po.thin3d)(a)[0]
        line = (po.centerline2d if flat else po.centerline3d)(a, 4, 2)
        for dtype in ("uint8", "int16", "float32"):
            v = a.astype(dtype)
            if pinned:
                v = torch.from_numpy(v).pin_memory().numpy()
            assert np.array_equal((Thinning2D if flat else Thinning3D)(v, ctx), want.astype(dtype))
            got = CenterlineExtraction(v, 4, 2, ctx)
            for g, w in zip(got, (line.x, line.y, *([] if flat else [line.z]), line.idx), strict=True):
                assert np.array_equal(g, w)


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
def test_routes(ctx, pinned):
    _check(ctx, pinned)


@pytest.mark.gpu
def test_routes_on_one_cpu(ctx):
    _one_cpu("from begputhinning_b200 import Context\nfrom tests.test_host_route import _check\nc = Context(0)\n"
             "_check(c, False)\n_check(c, True)\nc.close()")
