"""A context on a second GPU, after the first one was used: kernels with more than 48 KB
of shared memory are opted in on each device."""
import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def test_crowded_scene_on_each_device(cb):
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    a = O.aabb(S.clustered_spheres(12_000, seed=3, clusters=2, sigma=0.01, background=0.05))
    _, p = O.broadphase(a, (32, 32, 32))
    for dev in (0, 1):
        with torch.cuda.device(dev):
            bp = cb.Broadphase(cb.Context(dev))
            for _ in range(3):
                assert np.array_equal(bp.detectPossibleCollisions(torch.from_numpy(a.copy()).cuda()).cpu().numpy(), p)
