"""A pair list retained after CC_ERR_CAPACITY (cc_broadphase_fetch) is the whole
list, whatever the context computed in between."""
import ctypes
import os
import subprocess
import sys

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


def lattice(n, moved):
    """n unit-spaced spheres; the first `moved` of every second body touch their neighbour."""
    k = int(np.ceil(n ** (1 / 3)))
    c = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n].astype(np.float32)
    c[0:2 * moved:2] = c[1:2 * moved:2] + np.float32(0.125)
    B = np.zeros((n, 3), np.float32)
    B[:, 0] = 0.25
    return S._one_shape_per_body(np.full(n, S.SPHERE), B, c, S._identity_quats(n), "lattice")


def short_list_fetched(cb, n, cap=16, moved=600):
    """cc_collide on a scene without a pair, then with `moved` of them and no room, then the fetch."""
    still, touching = lattice(n, 0), lattice(n, moved)
    _, p = O.broadphase(O.aabb(touching), (32, 32, 32))
    assert len(p) >= moved
    ds, ctx = cb.DeviceScene(still), cb.Context()
    pipe = cb.DevicePipeline(ds, ctx=ctx, pairs_cap=cap)
    for _ in range(2):
        ds.pos.copy_(torch.from_numpy(still.pos))
        assert pipe.run() == (0, 0)
        ds.pos.copy_(torch.from_numpy(touching.pos))
        st = _lib.lib.cc_collide(ctx.h, ctypes.byref(pipe.scene), 16, 16, 16, 0.0, ctypes.byref(pipe.res), None)
        assert st == _lib.CC_ERR_CAPACITY and pipe.res.n_pairs == len(p)
        assert np.array_equal(fetch(ctx, len(p)), p)


@pytest.mark.parametrize("n", [1500, 9000, 300_001])
def test_short_list(cb, n):
    # above 262,144 bodies the last call's empty list leaves too many owner buckets for the one-launch sort
    short_list_fetched(cb, n)


def test_short_list_without_the_fused_sort():
    env = dict(os.environ, CC_FUSED_SORT="0")
    code = "import conftest, collide_b200 as cb, test_gpu_fetch as t; t.short_list_fetched(cb, 9000); t.short_list_fetched(cb, 1500)"
    subprocess.run([sys.executable, "-c", code], check=True, env=env, cwd=os.path.dirname(os.path.abspath(__file__)))
