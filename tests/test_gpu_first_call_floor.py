"""The first call of a new context on a scene with a body over many search cells and no
crowded one: the search is done again on sorted cells, without the dense-cell test."""
import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2_500, 6_000, 70_000])
def test_second_search_is_the_plain_one(cb, n):
    edge = (n * 1e-5) ** (1 / 3)  # 0.2 pairs a body and those of the floor: within the first guess
    a = O.aabb(S.spheres_uniform(n, seed=n, hi=edge))
    a[n - 1], a[-1] = (0.0, 0.0, -0.01), (edge, edge, 0.001)
    _, p = O.broadphase(a, (16, 16, 16))
    assert len(p) < n // 4 + 1024
    boxes, ctx, launches = torch.from_numpy(a).cuda(), cb.Context(), []
    bp = cb.Broadphase(ctx)
    bp.number_of_contacts_possible = len(p)  # room for the list at once
    for _ in range(3):
        assert np.array_equal(bp.detectPossibleCollisions(boxes.clone()).cpu().numpy(), p)
        launches.append(ctx.launches())
    assert launches[0] <= launches[2] + 5, launches  # link, check, walk, a sort that had nothing, another grid
