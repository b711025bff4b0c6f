"""A CPU model of the protocol by which the boxes of a volume thin it together
(begputhinning_b200/csrc/resident.cu: res_run3d): boxes of rows and planes at
full width with six halo rows and planes, words of 30 voxels, a list of the
words that are non-empty at the start and at most five rows or planes from the
core, words looked at only when a word of the rows around them changed in the
previous iteration (at the granularity of the rows' eight mask columns),
subiteration J leaving words alone that are farther than 5 - J from the core,
and after every iteration the changed words near a core's edge taken over by
the boxes around it.  Deletions use the oracle's rule tables.  The model must
reproduce the oracle, one word per row included, and must fail with a halo too
small and with the row of a word taken from a reciprocal that does not hold."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.helpers import blobs3d

OFFS = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dz, dy, dx) != (0, 0, 0)]
TABLES = [po.rule_table(3, d) for d in range(6)]  # 2^21 words: bit n % 32 of word n / 32 = deletable


def deletable(v, d):
    p = np.pad(v, 1)
    n = np.zeros(v.shape, np.int64)
    for i, (dz, dy, dx) in enumerate(OFFS):
        n |= p[1 + dz:p.shape[0] - 1 + dz, 1 + dy:p.shape[1] - 1 + dy, 1 + dx:p.shape[2] - 1 + dx].astype(np.int64) << i
    return ((TABLES[d][n >> 5] >> (n & 31).astype(np.uint32)) & 1).astype(bool) & (v != 0)


def per_word(m):
    """Whether a word of 30 voxels has any."""
    wl = -(-m.shape[2] // 30)
    p = np.zeros((*m.shape[:2], 30 * wl), bool)
    p[:, :, :m.shape[2]] = m
    return p.reshape(*m.shape[:2], wl, 30).any(3)


def per_voxel(words, width):
    return np.repeat(words, 30, 2)[:, :, :width]


def row_by_reciprocal(rest, p):
    """As the kernel divides: exact for a pitch of one as well."""
    return (2 * rest * (0x7FFFFFFF // p + 1)) >> 32


def row_by_wrapping_reciprocal(rest, p):
    """2^32 / p in 32 bits: none for a pitch of one."""
    return (rest * ((0xFFFFFFFF // p + 1) & 0xFFFFFFFF)) >> 32


class Box:
    def __init__(self, vol, z, y, halo, row_of):
        D, H, W = vol.shape
        (self.r0, self.r1), (self.c0, self.c1) = z, y
        self.z0, self.z1 = max(0, self.r0 - halo), min(D, self.r1 + halo)
        self.y0, self.y1 = max(0, self.c0 - halo), min(H, self.c1 + halo)
        self.v = vol[self.z0:self.z1, self.y0:self.y1].copy()
        self.wl = -(-W // 30)
        self.xs = 0
        while (self.wl - 1) >> self.xs > 7:
            self.xs += 1
        zz, yy = np.mgrid[self.z0:self.z1, self.y0:self.y1]
        self.dist = np.maximum.reduce([self.c0 - yy, yy - self.c1 + 1, self.r0 - zz, zz - self.r1 + 1, 0 * zz])[:, :, None]
        self.listed = per_word(self.v != 0) & (self.dist <= 5)
        # the row (padding included) that a word's mask is looked up and marked at
        p = self.wl | 1
        y2 = np.arange(1, self.v.shape[1] + 1)[None, :, None] * p + np.arange(self.wl)[None, None, :]
        self.row = row_of(np.broadcast_to(y2, self.listed.shape).astype(object), p).astype(int)
        self.masks = np.ones((self.v.shape[0] + 2, self.v.shape[1] + 2, 8), bool)
        self.marks = np.zeros_like(self.masks)

    def mark(self, words):
        for z, y, w in np.argwhere(words):
            self.marks[z + 1, self.row[z, y, w], w >> self.xs] = True

    def iterate(self):
        z, y, w = np.nonzero(self.listed)
        active = np.zeros_like(self.listed)
        active[z, y, w] = self.masks[z + 1, self.row[z, y, w], w >> self.xs]
        W = self.v.shape[2]
        union = np.zeros(self.v.shape, bool)
        for d in range(6):
            union |= deletable(self.v, d)
        union &= per_voxel(active, W)
        before = self.v
        for j in range(6):
            self.v = np.where(deletable(self.v, j) & union & per_voxel(np.broadcast_to(self.dist <= 5 - j, self.listed.shape), W),
                              0, self.v).astype(np.uint8)
        changed = per_word(self.v != before) & (self.dist == 0)
        self.mark(changed)
        return changed

    def sent(self, changed, shape, halo):
        """Changed words near an edge of the core that another box may hold: (z, y, word, voxels)."""
        D, H, W = shape
        out = []
        for z, y, w in np.argwhere(changed):
            gz, gy = z + self.z0, int(self.row[z, y, w]) + self.y0 - 1
            if ((self.r0 > 0 and gz < self.r0 + halo) or (self.r1 < D and gz >= self.r1 - halo)
                    or (self.c0 > 0 and gy < self.c0 + halo) or (self.c1 < H and gy >= self.c1 - halo)):
                out.append((gz, y + self.y0, w, self.v[z, y, 30 * w:30 * w + 30].copy()))
        return out

    def take(self, msgs):
        for z, y, w, voxels in msgs:
            if self.z0 <= z < self.z1 and self.y0 <= y < self.y1:
                self.v[z - self.z0, y - self.y0, 30 * w:30 * w + 30] &= voxels
                self.marks[z - self.z0 + 1, y - self.y0 + 1, w >> self.xs] = True

    def next_masks(self):
        p = np.pad(self.marks, 1)
        m = np.zeros_like(self.marks)
        for dz in range(3):
            for dy in range(3):
                for dx in range(3):
                    m |= p[dz:dz + m.shape[0], dy:dy + m.shape[1], dx:dx + m.shape[2]]
        self.masks = m
        self.marks = np.zeros_like(m)


def run_boxes(vol, gz, gy, halo=6, row_of=row_by_reciprocal):
    D, H, W = vol.shape
    cut = halo if gz * gy > 1 else 0
    boxes = [Box(vol, (k * D // gz, (k + 1) * D // gz), (j * H // gy, (j + 1) * H // gy), cut, row_of)
             for k in range(gz) for j in range(gy)]
    for _ in range(200):
        changed = [b.iterate() for b in boxes]
        if not any(c.any() for c in changed):
            break
        msgs = [b.sent(c, vol.shape, halo) for b, c in zip(boxes, changed)]
        for i, b in enumerate(boxes):
            kz, ky = divmod(i, gy)
            for k in range(max(0, kz - 1), min(gz, kz + 2)):
                for j in range(max(0, ky - 1), min(gy, ky + 2)):
                    if (k, j) != (kz, ky):
                        b.take(msgs[k * gy + j])
            b.next_masks()
    out = np.zeros_like(vol)
    for b in boxes:
        out[b.r0:b.r1, b.c0:b.c1] = b.v[b.r0 - b.z0:b.r1 - b.z0, b.c0 - b.y0:b.c1 - b.y0]
    return out


def _volumes(shape):
    rng = np.random.default_rng(sum(shape))
    return [blobs3d(rng, *shape, max(4, np.prod(shape) // 1500), rmax=8), (rng.random(shape) < 0.5).astype(np.uint8),
            np.ones(shape, np.uint8)]


SHAPES = [((26, 30, 30), 2, 2), ((13, 40, 24), 1, 3), ((40, 12, 1), 3, 1), ((20, 24, 31), 2, 2), ((12, 26, 65), 1, 2),
          ((18, 14, 270), 2, 1), ((14, 15, 9), 1, 1)]


@pytest.mark.parametrize("shape,gz,gy", SHAPES)
def test_boxes_match_the_oracle(shape, gz, gy):
    for vol in _volumes(shape):
        assert np.array_equal(run_boxes(vol, gz, gy), po.thin3d(vol)[0])


@pytest.mark.parametrize("wrong", [dict(halo=0), dict(row_of=row_by_wrapping_reciprocal)])
def test_model_tells_a_broken_protocol(wrong):
    differ = [not np.array_equal(run_boxes(vol, gz, gy, **wrong), po.thin3d(vol)[0])
              for shape, gz, gy in SHAPES[:2] for vol in _volumes(shape)]
    assert any(differ)


def test_reciprocals():
    n = np.arange(1 << 16, dtype=np.uint64)
    for d in [*range(1, 400), 1023, 1024, 4097, 21845, 32767, 32768]:
        assert np.array_equal((2 * n * np.uint64(0x7FFFFFFF // d + 1)) >> np.uint64(32), n // np.uint64(d))
