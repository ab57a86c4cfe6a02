"""A pair list retained after CC_ERR_CAPACITY (cc_broadphase_fetch) is the whole
list, whatever the context computed in between."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import _lib
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def broadphase_too_small(cb, ctx, boxes, cap=16):
    t = torch.from_numpy(boxes.copy()).cuda()
    out = torch.empty(cap, dtype=torch.int64, device="cuda")
    n = ctypes.c_uint64()
    st = _lib.lib.cc_broadphase(ctx.h, boxes.shape[0] // 2, t.data_ptr(), 16, 16, 16, out.data_ptr(), cap,
                                ctypes.byref(n), None)
    assert st == _lib.CC_ERR_CAPACITY
    return n.value


def fetch(ctx, n):
    out = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    assert _lib.lib.cc_broadphase_fetch(ctx.h, out.data_ptr(), n, None) == _lib.CC_OK
    return out.cpu().numpy()


@pytest.mark.parametrize("crowded", [True, False])
def test_a_narrowphase_in_between(cb, crowded):
    sc = S.clustered_spheres(12_000, seed=3, clusters=2, sigma=0.01, background=0.05) if crowded else \
        S.mixed_slab(12_000, seed=3, extent=(0.4, 0.4, 0.1))
    other = cb.DeviceScene(S.mixed_slab(900, seed=4, extent=(0.1, 0.1, 0.05)))
    boxes = O.aabb(sc)
    _, p = O.broadphase(boxes, (32, 32, 32))
    q = torch.from_numpy(np.stack([np.arange(0, 800, 2), np.arange(1, 801, 2)])).cuda()
    ctx = cb.Context()
    for _ in range(3):  # found out by the chains, tested twice, masks kept
        assert broadphase_too_small(cb, ctx, boxes) == len(p)
        cb.Narrowphase(ctx).DoNarrowphase(other.T, other.A, other.B, other.C, other.R, other.ID, other.active, other.pos,
                                          other.rot, (q[0] << 32) | q[1])
        assert np.array_equal(fetch(ctx, len(p)), p)
