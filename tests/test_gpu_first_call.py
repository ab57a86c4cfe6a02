"""The first call of a new context, which knows nothing of its scene: boxes that lie
in more than three search cells each (the most that cells of two mean extents give is
1.5^3) need no second search."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [40, 48, 101])
def test_no_second_search(cb, k):
    # boxes of 0.49 spacings jittered on a lattice, cells that sweep over them: 1.48^3 = 3.2 cells each, no pair
    rng = np.random.default_rng(k)
    lo = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    lo = (lo + rng.uniform(0.0, 0.5, lo.shape)).astype(np.float32)
    boxes = torch.from_numpy(np.concatenate([lo, lo + np.float32(0.49)])).cuda()
    ctx = cb.Context()
    ctx.set_search_grid((k - 1, k - 1, k - 1))
    bp, launches = cb.Broadphase(ctx), []
    for _ in range(2):
        assert bp.detectPossibleCollisions(boxes.clone()).numel() == 0
        launches.append(ctx.launches())
    assert launches[0] == launches[1] + 1  # the look for crowded cells
