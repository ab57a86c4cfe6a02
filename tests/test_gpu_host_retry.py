"""A host step whose pair list does not fit leaves the caller's arrays alone, the box
array above all: it holds the boxes of RECT and TRIANGLEMESH shapes, which the
caller's next try starts from."""
import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
def test_boxes_kept_for_the_next_try(cb, pinned):
    # 2,100 boxes of 0.75 search cells: 5.4 entries and 0.85 pairs a body. A first search with room
    # for 3.5 entries finds fewer pairs than there are, and these would fit the output.
    n, r = 2100, np.float32(0.375)
    rng = np.random.Generator(np.random.PCG64(2))
    pos = rng.uniform(-8.0, 8.0, (n, 3)).astype(np.float32)
    T = np.where(rng.random(n) < 0.3, S.RECT, S.SPHERE).astype(np.int32)
    B = np.zeros((n, 3), np.float32)
    B[:, 0] = r
    B[T == S.RECT, 1] = r
    sc = S._one_shape_per_body(T, B, pos, S._identity_quats(n), "plates")
    boxes = np.concatenate([pos - r, pos + r])
    shifted, p = O.broadphase(boxes, (16, 16, 16))
    given = boxes.copy()
    given[np.tile(T == S.SPHERE, 2)] = 7.0  # GenerateAABB writes these
    ctx = cb.Context()
    ctx.set_search_grid((16, 16, 16))
    s = cb.HostSession(sc, ctx=ctx, want_aabb=True, pinned=pinned, pairs_cap=len(p) - len(p) // 16)
    s.aabb.copy_(torch.from_numpy(given))
    s.pairs.fill_(-5)
    kept, tries = s._alloc, []

    def grown(cap):
        assert np.array_equal(s.aabb.numpy(), given) and bool((s.pairs == -5).all())
        tries.append(cap)
        kept(cap)

    s._alloc = grown
    P, _ = s.run()
    assert len(tries) == 1 and P == len(p) and np.array_equal(np.sort(s.pairs[:P].numpy()), p)
    assert np.array_equal(s.aabb.numpy(), shifted)
