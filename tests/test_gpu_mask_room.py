"""Hit masks of crowded cells are optional scratch: a device short of memory gives
them less room, or none, and the call still returns the whole pair list."""
import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def test_little_free_memory(cb):
    n = 150_000  # all of them in the one cell of a pinned grid: 1.4 GB of masks
    a = O.aabb(S.spheres_uniform(n, seed=8))
    _, p = O.broadphase(a, (32, 32, 32))
    ctx = cb.Context()
    ctx.set_search_grid((1, 1, 1))
    bp, boxes = cb.Broadphase(ctx), torch.from_numpy(a).cuda()
    for free in (None, 0.8, 0.8, 0.1):  # GB left; the first call makes no masks
        held = None
        if free is not None:
            torch.cuda.empty_cache()
            held = torch.empty(torch.cuda.mem_get_info()[0] - int(free * 2 ** 30), dtype=torch.uint8, device="cuda")
        assert np.array_equal(bp.detectPossibleCollisions(boxes.clone()).cpu().numpy(), p), free
        del held
    torch.cuda.empty_cache()
    for _ in range(40):  # and with room again, until they are asked for once more
        got = bp.detectPossibleCollisions(boxes.clone())
    assert np.array_equal(got.cpu().numpy(), p)
