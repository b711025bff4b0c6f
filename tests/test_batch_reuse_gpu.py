"""A batch laid out again in its reserved memory."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po
from tests.helpers import blobs3d, random2d

pytestmark = pytest.mark.gpu


def _add(b, items):
    return [b.add(v.shape) for v in items]


def _run(b, ids, items):
    import torch
    ins = [torch.from_numpy(v).cuda() for v in items]
    outs = [torch.full_like(t, 7) for t in ins]
    for i, t, o in zip(ids, ins, outs):
        b.set_io(i, t, o)
    b.run()
    for v, o in zip(items, outs):
        assert np.array_equal(o.cpu().numpy(), (po.thin2d if v.ndim == 2 else po.thin3d)(v)[0])


def test_no_records_before_a_run(ctx):
    from begputhinning_b200 import Batch, lib
    rng = np.random.default_rng(2)
    items = [random2d(rng, 90, 200, 0.5), blobs3d(rng, 30, 40, 50, 6)]
    b = Batch(ctx)
    try:
        assert lib().bgt_batch_reserve(b.h, C.c_size_t(64 << 20)) == 0
        for _ in range(2):
            ids = _add(b, items)
            b.finalize()
            for i in ids:
                s = b.stats(i)
                assert (s["passes"], s["converged"]) == (0, 0)
            assert b.work() == (0, 0)
            _run(b, ids, items)
            assert all(b.stats(i)["converged"] == 1 and b.stats(i)["passes"] > 0 for i in ids)
            assert lib().bgt_batch_reset(b.h) == 0
    finally:
        b.close()


def test_pools_too_small_for_messages(ctx):
    """Reserved memory that holds the tile rings' plan takes the instances,
    whichever engine then thins them."""
    from begputhinning_b200 import Batch, lib
    rng = np.random.default_rng(3)
    items = [blobs3d(rng, 90, 100, 110, 30, rmax=9), blobs3d(rng, 20, 30, 40, 4)]
    items += [random2d(rng, 80, 70 + k, 0.5) for k in range(12)]
    rest = len(items) - 1

    def sized(rings):
        b = Batch(ctx)
        b.set_engine(rings)
        ids = _add(b, items)
        b.finalize()
        plan = [b.plan(i) for i in ids]
        n = b.device_bytes()
        b.close()
        return n, plan

    (rings, _), (boxes, plan) = sized(True), sized(False)
    assert plan[0][1] > 1 and boxes > rings + (1 << 20)
    for reserved, resident in ((boxes, [True] * (rest + 1)), (rings + 8192, [False] + [True] * rest),
                               (rings, [False] * (rest + 1))):
        b = Batch(ctx)
        try:
            assert lib().bgt_batch_reserve(b.h, C.c_size_t(reserved)) == 0
            ids = _add(b, items)
            b.finalize()
            assert [b.plan(i)[0] for i in ids] == resident
            _run(b, ids, items)
            assert lib().bgt_batch_reset(b.h) == 0
        finally:
            b.close()
