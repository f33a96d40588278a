"""The rule by which an RK stage of the BSSN evolution writes its neighbours' ghost layers (EvoArgs::feed,
evolve_sim.cu, kernels_evolve_stage.cu), on the CPU: on random sets of same-depth domains, with and
without periodic faces, the fed cells and the fill's remaining faces give every cell the value of the plain fill."""
from __future__ import annotations

import itertools

import numpy as np
import pytest

N, P = 8, 3
T = N + 2 * P


def face(axis, side, ghost):
    """The cells of a face's ghost layers (side 0: +), or of its same-depth source; array order z, y, x."""
    at = [None] * 3
    for b in range(3):
        if b == axis:
            at[2 - b] = (slice(P + N, T) if side == 0 else slice(0, P)) if ghost else (slice(P, 2 * P) if side == 0 else slice(N, N + P))
        else:
            at[2 - b] = slice(0, T) if b < axis else slice(P, P + N)
    return tuple(at)


def fill(x, source, skip):
    """Three passes: the copies not in `skip`, and a stand-in for the interpolated faces."""
    for a in range(3):
        y = x.copy()
        for (i, b, s), j in source.items():
            if b == a and j >= 0 and (i, a, s) not in skip:
                y[(i,) + face(a, s, True)] = x[(j,) + face(a, s, False)]
            elif b == a and j < 0:
                v = y[(i,) + face(a, s, True)]
                y[(i,) + face(a, s, True)] = 1000 * i + 10 * a + s + np.arange(v.size).reshape(v.shape) * 1e-4
        x = y
    return x


@pytest.mark.parametrize("axes", [2, 3])
@pytest.mark.parametrize("periodic,seed", [(True, 1), (True, 2), (False, 3), (False, 4)])
def test_fed_cells_equal_the_fill(periodic, seed, axes):
    rng = np.random.default_rng(seed)
    cells = [c for c in itertools.product(range(3), repeat=3) if rng.random() < .8]
    slot = {c: i for i, c in enumerate(cells)}
    source = {}
    for c, i in slot.items():
        for a, s in itertools.product(range(3), range(2)):
            q = list(c)
            q[a] += 1 if s == 0 else -1
            if periodic:
                q[a] %= 3
            source[i, a, s] = slot.get(tuple(q), -1)
    x = rng.random((len(cells), T, T, T))
    feed, fed = {}, set()
    for a in range(axes):
        for (i, b, s), j in sorted(source.items()):
            if b == a and j >= 0 and (j, a, s) not in feed and all((j, e, q) in fed for e in range(a) for q in range(2)):
                feed[j, a, s] = i
                fed.add((i, a, s))
    y = x.copy()

    def image(at, axis, w):   # of a cell, in the next domain along the axis
        s = 0 if w < P else (1 if w >= N - P else -1)
        if at is None or s < 0 or (at[0], axis, s) not in feed:
            return None
        q = list(at)
        q[0] = feed[at[0], axis, s]
        q[3 - axis] += N if s == 0 else -N
        return tuple(q)

    for i in range(len(cells)):
        for k, j, h in itertools.product(range(N), repeat=3):
            own = (i, k + P, j + P, h + P)
            gx, gy, gz = image(own, 0, h), image(own, 1, j), image(own, 2, k)
            gxy = image(gx, 1, j)
            for at in (gx, gy, gz, gxy, image(gx, 2, k), image(gy, 2, k), image(gxy, 2, k)):
                if at is not None:
                    y[at] = x[own]
    assert fed and np.array_equal(fill(y, source, fed), fill(x, source, set()))
