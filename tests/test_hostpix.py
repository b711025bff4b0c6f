"""CPU: the host's pixel packing (begputhinning_b200/csrc/hostpix.cpp) against
the oracle's binarisation for every pixel type and rule, at word edges, padded
extents and sizes that take several parts, alone and on the worker threads;
and the way back."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po

CODES = {"uint8": 0, "int8": 1, "uint16": 3, "int16": 4, "uint32": 5, "int32": 6, "float32": 7, "float64": 8, "bool": 9}


@pytest.fixture(scope="module", params=[False, True], ids=["alone", "workers"])
def L(request):
    from begputhinning_b200 import lib
    h = lib()
    if request.param:
        h._ZN3bgt16host_pool_retainEv()
    yield h
    if request.param:
        h._ZN3bgt17host_pool_releaseEv()


def _values(rng, shape, dtype):
    if dtype.startswith("f"):
        v = rng.choice([0.0, -0.0, 0.25, 0.999, 1.0, 1.5, -1.0, -3.5, 2147483520.0, 2147483648.0, 5e9, -5e9, np.inf, -np.inf,
                        np.nan], shape)
        return v.astype(dtype)
    if dtype == "bool":
        return rng.random(shape) < 0.5
    info = np.iinfo(dtype)
    edge = [0, 1, 2, info.min, info.max, info.max // 2, info.max // 2 + 1, max(info.min, -1)]
    return rng.choice(np.array(edge, dtype), shape)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("dtype", list(CODES))
@pytest.mark.parametrize("shape", [(1, 1), (3, 31), (5, 32), (7, 33), (64, 100), (700, 1031), (2, 3, 65), (40, 70, 300)])
def test_pack_and_unpack(L, dtype, shape):
    rng = np.random.default_rng(sum(shape))
    a = _values(rng, shape, dtype)
    d, h, w = (1, *shape) if len(shape) == 2 else shape
    H, D, P = h + 5, d + (len(shape) == 3), ((w + 31) // 32 + 3) // 4 * 4 + 4
    words = np.full((D, H, P), 0xDEADBEEF, np.uint32)
    L._ZN3bgt9host_packEiiPKviiiiiiPj(CODES[dtype], 0 if len(shape) == 2 else 1, _ptr(a), w, h, d, H, D, P, _ptr(words))
    bits = np.unpackbits(words.view(np.uint8), bitorder="little").reshape(D, H, 32 * P)
    want = po.binarise(a, CODES[dtype], len(shape)).reshape(d, h, w)
    assert np.array_equal(bits[:d, :h, :w], want)
    assert bits.sum() == want.sum()  # nothing outside the array

    back = np.full((d, h, w), 7).astype(dtype)
    rows = np.ascontiguousarray(words[:d, :h])
    L._ZN3bgt11host_unpackEiPKjiiiiPv(CODES[dtype], _ptr(rows), w, h, d, P, _ptr(back))
    assert np.array_equal(back, want.astype(dtype))
