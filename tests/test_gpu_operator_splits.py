"""The single-operator stencils' even split of planes over the grid, and the criterion's octants, against
the same operators on fewer domains, whose launch splits the planes at other places."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,used", [(8, 2, 1), (8, 2, 37), (16, 3, 1), (16, 3, 151), (28, 2, 49), (28, 2, 151), (32, 3, 5),
                                      (32, 3, 153)])
def test_operators_equal_domain_by_domain(am, cuda, n, p, used):
    """Words and criterion values of `used` domains (dead ones among them) equal those of a launch over the
    domains up to one of them with only that one alive, bit for bit: a cell's arithmetic and noise depend on
    its domain and place alone."""
    import torch
    from adaptivemesh_gb300 import ops
    cfg, t = am.Config(n, p, 10.0), n + 2 * p
    g = torch.Generator(device="cuda").manual_seed(n + used)
    field = torch.randn(used * t ** 3, generator=g, device="cuda", dtype=torch.float32)
    new = lambda *s: torch.zeros(s, dtype=torch.int32, device="cuda")  # noqa: E731
    # positions: depth in the top bits as the octree packs it; every third slot dead
    pos = np.array([0xFFFFFFFF if s % 3 == 2 else (s % 3) << 27 for s in range(used)], np.uint32)

    def run(positions):
        used = len(positions)
        dpos = torch.from_numpy(positions.view(np.int32)).cuda()
        dif, d2, off = new(used * n ** 3), new(used * n ** 3), new(used * n ** 3)
        crit = torch.zeros(used * n * n, dtype=torch.float32, device="cuda")
        ops.differentiate(cfg, field, dif, d2, dpos, used, 0, 4, 77)
        ops.mixed_partials(cfg, field, off, dpos, used, 0, 4, 78)
        ops.criterion(cfg, dif, d2, crit, dpos, used, 0, 4)
        torch.cuda.synchronize()
        return [x.cpu().numpy().reshape(used, -1) for x in (dif, d2, off, crit)]

    whole = run(pos)
    for s in sorted({0, 1, used // 2, used - 1} & set(range(used))):
        alone = np.full(s + 1, 0xFFFFFFFF, np.uint32)
        alone[s] = pos[s]
        for a, b, name in zip(whole, run(alone), ("gradient", "hessian", "mixed", "criterion")):
            assert np.array_equal(a[s].view(np.uint32), b[s].view(np.uint32)), (name, s)
    for s in range(used):   # dead slots are left alone, their criterion is NaN
        if pos[s] == 0xFFFFFFFF:
            assert all(not w[s].any() for w in whole[:3]) and np.isnan(whole[3][s]).all()
