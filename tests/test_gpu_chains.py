"""The chained search (cells as linked lists, taken while no cell is crowded)
where it can go wrong: block and warp edges of the body count, boxes over many
cells, a cell past the length at which the walk gives up, and the changes
between chained and sorted cells on one context. Pairs and shifted boxes equal
the oracle's, bit for bit, on every call."""
import numpy as np
import pytest
import torch

import oracle as O
from _helpers import same_bits
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def calls(cb, boxes, times=1, ctx=None):
    """`times` calls on one context for each array of boxes, all checked."""
    ctx = ctx or cb.Context()
    bp = cb.Broadphase(ctx)
    for a in boxes:
        sh, p = O.broadphase(a, (16, 16, 16))
        for _ in range(times):
            t = torch.from_numpy(a.copy()).cuda()
            got = bp.detectPossibleCollisions(t).cpu().numpy()
            assert np.array_equal(got, p)
            assert same_bits(t.cpu().numpy(), sh)
    return ctx


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 256, 257, 1023, 4097])
def test_body_counts(cb, n):
    calls(cb, [O.aabb(S.spheres_uniform(n, seed=n, hi=(n * 2e-6) ** (1 / 3)))], times=3)


@pytest.mark.parametrize("half", [0.004, 0.05, 0.2, 0.5])
def test_boxes_over_many_cells(cb, half):
    # a floor and a few large boxes over up to every cell of the grid (the largest: more than 65,535 cells)
    n = 120_000
    a = O.aabb(S.spheres_uniform(n, seed=1, rmin=0.001, rmax=0.002))
    rng = np.random.Generator(np.random.PCG64(2))
    big = rng.choice(n, 5, replace=False)
    a[big] = np.float32(0.5 - half)
    a[big + n] = np.float32(0.5 + half)
    a[big[0], :2], a[big[0] + n, :2] = 0.0, 1.0
    a[big[0], 2], a[big[0] + n, 2] = -0.01, 0.01
    calls(cb, [a], times=3)


@pytest.mark.parametrize("k", [100, 127, 128, 129, 130, 4095, 4096, 4097, 4200])
def test_long_chains_on_a_context_that_saw_none(cb, k):
    sparse = O.aabb(S.spheres_uniform(16384, seed=0))
    knot = sparse.copy()
    knot[:k], knot[16384:16384 + k] = np.float32(0.5), np.float32(0.50001)  # k boxes in one place
    calls(cb, [sparse, sparse, knot, knot, sparse, sparse, knot])


def test_fresh_context_meets_a_crowded_scene(cb):
    dense = O.aabb(S.clustered_spheres(60_000, seed=2, clusters=2, sigma=0.01, background=0.05))
    ctx = cb.Context()
    ctx.set_dense_cell(0)  # sorted cells, none of them dense: the chains are tried again in between
    calls(cb, [dense], times=40, ctx=ctx)
