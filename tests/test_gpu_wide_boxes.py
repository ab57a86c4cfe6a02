"""A body over many search cells (a floor, a boulder) sends its scene to sorted
cells, four times as large as chained ones, and keeps it there; without it the
context returns to chained cells. Pairs equal the oracle's on every call."""
import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def grid_of(cb, ctx, a, p):
    got = cb.Broadphase(ctx).detectPossibleCollisions(torch.from_numpy(a.copy()).cuda())
    assert np.array_equal(got.cpu().numpy(), p)
    return int(np.prod(ctx.last_grid()[0]))


@pytest.mark.parametrize("n", [6_000, 70_000])
@pytest.mark.parametrize("index", [0, -1])
def test_floor_comes_and_goes(cb, n, index):
    edge = (n * 4e-6) ** (1 / 3)
    a = O.aabb(S.spheres_uniform(n, seed=n, hi=edge))
    floor = a.copy()
    i = index % n
    floor[i], floor[n + i] = (0.0, 0.0, -0.01), (edge, edge, 0.001)
    (_, p), (_, q) = O.broadphase(a, (16, 16, 16)), O.broadphase(floor, (16, 16, 16))
    ctx = cb.Context()
    for _ in range(2):
        assert grid_of(cb, ctx, a, p) > n / 2           # a cell or more a body
    grid_of(cb, ctx, floor, q)                          # found out on chained cells, searched again
    for call in range(70):
        assert grid_of(cb, ctx, floor, q) < n / 2, call  # a cell for four bodies: never back on chains
    for call in range(40):
        last = grid_of(cb, ctx, a, p)
    assert last > n / 2


@pytest.mark.parametrize("cells,chained", [(2, True), (4, True), (9, False)])
def test_boulder(cb, cells, chained):
    # a cube over about cells^3 chained cells (one a body) at the end of the list
    n = 40_000
    edge = (n * 4e-6) ** (1 / 3)
    a = O.aabb(S.spheres_uniform(n, seed=1, hi=edge))
    half = np.float32(0.5 * cells * edge / n ** (1 / 3))
    a[n - 1], a[-1] = edge / 2 - half, edge / 2 + half
    _, p = O.broadphase(a, (16, 16, 16))
    ctx = cb.Context()
    for _ in range(3):
        last = grid_of(cb, ctx, a, p)
    assert (last > n / 2) == chained
