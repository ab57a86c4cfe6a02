"""Scenes with nearly as many owner buckets as the one-launch owner sort takes (8,191):
its offsets, keys and static words together need more than 48 KB of shared memory."""
import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


# ten pairs a body: one owner a bucket; a quarter of a pair: 32
@pytest.mark.parametrize("n,pairs", [(8_090, 10.0), (8_110, 10.0), (8_112, 10.0), (8_150, 10.0), (8_191, 10.0), (8_192, 10.0),
                                     (259_600, 0.25), (262_112, 0.25)])
def test_bucket_counts(cb, n, pairs):
    edge = (n * 0.0161 ** 3 / (2 * pairs)) ** (1 / 3)
    sc = S.spheres_uniform(n, seed=n, hi=edge)
    _, p = O.broadphase(O.aabb(sc), (24, 24, 24))
    pipe = cb.DevicePipeline(cb.DeviceScene(sc), ctx=cb.Context(), pairs_cap=2 * len(p))
    for _ in range(3):  # the buckets follow the last call's pairs
        P, C = pipe.run()
        keys = pipe.pairs[:P].cpu().numpy()
        assert P == len(p) and C > 0 and np.array_equal(np.sort(keys), p)
