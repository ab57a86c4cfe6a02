"""Small scenes, whose boxes are all tested against one another: pairs and shifted
boxes equal the oracle's bit for bit at the edges of the tiles, sparse and with
every box over every other, on both sides of the size where cells take over."""
import numpy as np
import pytest
import torch

import oracle as O
from _helpers import same_bits
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["sparse", "crowded", "knot"])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 255, 256, 257, 321, 1000, 2047, 2048, 2049])
def test_pairs(cb, n, kind):
    edge = (n * {"sparse": 2e-5, "crowded": 1e-6, "knot": 1e-12}[kind]) ** (1 / 3)
    a = O.aabb(S.spheres_uniform(n, seed=n, hi=edge))
    a -= np.float32(0.37)  # both signs: the shift is by |min|
    sh, p = O.broadphase(a, (4, 4, 4))
    bp = cb.Broadphase(cb.Context())
    for _ in range(3):  # the third call knows how many pairs there are
        t = torch.from_numpy(a.copy()).cuda()
        assert np.array_equal(bp.detectPossibleCollisions(t).cpu().numpy(), p)
        assert same_bits(t.cpu().numpy(), sh)


def test_invalid_boxes_change_nothing(cb):
    a = O.aabb(S.spheres_uniform(300, seed=1, hi=0.05))
    a[7, 1] = np.nan
    t = torch.from_numpy(a.copy()).cuda()
    with pytest.raises(Exception):
        cb.Broadphase(cb.Context()).detectPossibleCollisions(t)
    assert same_bits(t.cpu().numpy(), a)


def test_one_context_takes_small_and_large_scenes(cb):
    ctx = cb.Context()
    for n in (300, 5000, 2048, 2049, 40, 20_000, 1000):
        a = O.aabb(S.spheres_uniform(n, seed=n, hi=(n * 2e-6) ** (1 / 3)))
        sh, p = O.broadphase(a, (8, 8, 8))
        t = torch.from_numpy(a.copy()).cuda()
        assert np.array_equal(cb.Broadphase(ctx).detectPossibleCollisions(t).cpu().numpy(), p)
        assert same_bits(t.cpu().numpy(), sh)
