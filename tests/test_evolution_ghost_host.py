"""Host-side arithmetic of the evolution's ghost fill, checked on the CPU: the interpolating faces' source boxes
fit the shared memory that the kernel provides per axis at compile time (each extent at most half the filled
extent plus 5, the division of a box index by multiplication exact), on the trees of
test_evolution_host."""
from __future__ import annotations

import numpy as np
import pytest

from test_evolution_host import TREES, cases_cf3_decode


def box_extents(st, n, p=3):
    """(axis, per-axis source extents, per-axis filled extents) of every interpolating face, with the
    kernel's single-precision geometry."""
    f32, t = np.float32, n + 2 * p
    words = np.asarray(st["boundaries"], np.uint64)
    for slot in range(st["used_slots"]):
        if int(st["positions"][slot]) == 0xFFFFFFFF:
            continue
        for face in range(6):
            bd = int(words[slot * 6 + face])
            nd = bd & 0xFFFFFFFF
            cd, dd = nd >> 28, (nd >> 24) & 15
            if (nd & 0xFFFFFF) == 0xFFFFFF or cd in (0, 15) or dd == 0:
                continue
            rel, axis, side = cases_cf3_decode(bd >> 32), face % 3, face // 3
            root_src = (nd & 0xFFFFFF) == 0
            got, ext = [], []
            for a in range(3):
                lo = (p + n if side == 0 else 0) if a == axis else (0 if a < axis else p)
                ext.append(p if a == axis else (t if a < axis else n))
                w = np.arange(lo, lo + ext[a], dtype=np.float32)
                rp = ((w - f32(p) + f32(.5)) / f32(n) - f32(.5)) * (f32(1) / f32(1 << dd)) + f32(rel[a])
                ri = (rp + f32(.5)) * f32(n) + f32(p) - f32(.5)
                whole = root_src or a < axis
                b = np.clip(np.floor(ri).astype(np.int64), 1 if whole else p + 1, t - 3 if whole else t - p - 3)
                got.append(int(b[-1] - b[0] + 4))
            yield axis, got, ext


@pytest.mark.parametrize("tree", sorted(TREES))
@pytest.mark.parametrize("n", [8, 16, 32])
def test_source_boxes_fit_per_axis(am, tree, n):
    o = am.Octree(3000)
    TREES[tree](o)
    st = o.state()
    o.close()
    seen = 0
    for axis, got, ext in box_extents(st, n):
        assert all(g <= e // 2 + 5 for g, e in zip(got, ext)), (tree, n, axis, got, ext)
        size = got[0] * got[1] * got[2]
        e = np.arange(size, dtype=np.uint64)
        q = (e * np.uint64(((1 << 21) + got[0] - 1) // got[0])) >> np.uint64(21)
        assert np.array_equal(q, e // np.uint64(got[0]))
        assert np.array_equal((q * np.uint64(((1 << 21) + got[1] - 1) // got[1])) >> np.uint64(21), q // np.uint64(got[1]))
        seen += 1
    assert seen
