"""Incremental steps asked for the pair count alone (no output arrays), rebuild and
kept ones, then with room: counts and results equal those of full steps."""
import ctypes

import pytest
import torch

from collide_b200 import _lib
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1500, 30_011])
def test_count_then_step(cb, n):
    ds = cb.DeviceScene(S.mixed_slab(n, seed=n, extent=(0.6, 0.6, 0.1)))
    ref = cb.collide(ds, ctx=cb.Context())
    ctx = cb.Context()
    ctx.set_incremental(True, 1.0)
    aabb = torch.zeros((2 * n, 3), device="cuda")
    res = _lib.Result()
    res.aabb = aabb.data_ptr()
    sc = ds.c_scene()
    for step in range(3):
        st = _lib.lib.cc_collide(ctx.h, ctypes.byref(sc), 16, 16, 16, 0.0, ctypes.byref(res), None)
        assert st == _lib.CC_ERR_CAPACITY and res.n_pairs == ref["n_pairs"]
        assert ctx.last_step_rebuilt() == (step == 0)
        assert torch.equal(aabb, ref["aabb"])
    pipe = cb.DevicePipeline(ds, ctx=ctx, pairs_cap=ref["n_pairs"])
    for _ in range(2):
        assert pipe.run() == (ref["n_pairs"], ref["n_contacts"])
        assert torch.equal(pipe.pairs, ref["pairs"]) and torch.equal(pipe.norm[: ref["n_contacts"]], ref["norm"])
