"""The contact compaction (hit-first, stable) at its tile and grid edges: one row
a thread held in registers where a block's share is one tile, several tiles a
block beyond the co-resident grid, lists without and with only hits."""
import numpy as np
import pytest
import torch

from collide_b200 import scenes as S
from test_gpu_narrowphase import run_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("count", [1, 255, 256, 257, 5 * 148 * 256 - 1, 5 * 148 * 256 + 1, 8 * 148 * 256 + 257])
def test_results_in_order(cb, count, share):
    # spheres of radius 0.625 one apart: neighbours touch, next neighbours do not; every value is exact
    n = 1000
    B = np.zeros((n, 3))
    B[:, 0] = 0.625
    q = np.zeros((n, 4))
    q[:, 0] = 1.0
    pos = np.zeros((n, 3))
    pos[:, 0] = np.arange(n)
    m = S._one_shape_per_body(np.full(n, S.SPHERE, np.int32), B, pos, q, "row")
    rng = np.random.Generator(np.random.PCG64(count))
    i = rng.integers(0, n - 2, count)
    hit = rng.random(count) < share
    p = (i << 32) | (i + np.where(hit, 1, 2))
    got = run_np(cb, m, p.astype(np.int64))
    k = int(hit.sum())
    assert got["n"] == k
    assert np.array_equal(got["pairs"], np.concatenate([p[hit], p[~hit]]))
    assert np.array_equal(got["bids"][:k], np.stack([i[hit], i[hit] + 1], 1))
    x = np.array([1.0, 0.0, 0.0])
    assert np.array_equal(got["norm"][:k], np.broadcast_to(x, (k, 3)))
    assert np.array_equal(got["cpta"][:k], pos[i[hit]] + 0.625 * x)
    assert np.array_equal(got["cptb"][:k], pos[i[hit] + 1] - 0.625 * x)
    assert np.array_equal(got["depth"][:k], np.full(k, -0.25))


@pytest.mark.parametrize("n,extent", [(5_000, (0.3, 0.3, 0.1)), (60_000, (0.29, 0.29, 0.145))])
def test_results_by_the_hash(cb, n, extent):
    m = S.mixed_slab(n, seed=n, extent=extent)
    ref_ctx, ov_ctx = cb.Context(), cb.Context()
    ref_ctx.set_narrowphase_overlap(False)
    a = cb.DevicePipeline(cb.DeviceScene(m), ctx=ref_ctx, pairs_cap=6 * n)
    b = cb.DevicePipeline(cb.DeviceScene(m), ctx=ov_ctx, pairs_cap=6 * n)
    for step in range(4):
        P, C = a.run()
        assert b.run() == (P, C) and C > 0
        assert n < 60_000 or P > 5 * 148 * 256
        assert torch.equal(a.pairs[:P], b.pairs[:P]), step
        for k in ("norm", "cpta", "cptb", "depth", "bids"):
            assert torch.equal(getattr(a, k)[:C].view(torch.int32), getattr(b, k)[:C].view(torch.int32)), (step, k)
