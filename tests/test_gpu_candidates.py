"""The candidate filter of incremental steps at the edges of its tiles: kept steps
equal full searches bit for bit, from one candidate to several tiles of them, with
all, some and none of them overlapping."""
import numpy as np
import pytest
import torch

from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 1023, 1024, 1025, 1026, 2049, 40_000])
def test_kept_steps_equal_full_searches(cb, n):
    # a row of spheres of radius 0.52 one apart: n - 1 overlapping neighbours
    B = np.zeros((n, 3))
    B[:, 0] = 0.52
    q = np.zeros((n, 4))
    q[:, 0] = 1.0
    pos = np.zeros((n, 3))
    pos[:, 0] = np.arange(n) % 200
    pos[:, 1] = 3 * (np.arange(n) // 200)
    m = S._one_shape_per_body(np.full(n, S.SPHERE, np.int32), B, pos, q, "rows")
    full, inc = cb.Context(), cb.Context()
    inc.set_incremental(True, 0.3)
    a, b = cb.DevicePipeline(cb.DeviceScene(m), ctx=full, pairs_cap=2 * n), cb.DevicePipeline(cb.DeviceScene(m), ctx=inc, pairs_cap=2 * n)
    start = a.ds.pos.clone()
    rng = torch.Generator(device="cuda").manual_seed(n)
    seen = []
    for spread in (1.0, 1.0, 1.02, 1.0, 1.06, 1.03, 1.0):  # 1.04 and more pulls the row apart
        p = start.clone()
        near = torch.rand((n,), generator=rng, device="cuda") * 0.02
        p[:, 0] = (p[:, 0] - 100) * spread + 100 if n <= 3 else p[:, 0] + near * (spread - 0.97) / 0.03
        for x in (a, b):
            x.ds.pos.copy_(p)
        P, C = a.run()
        assert b.run() == (P, C)
        assert torch.equal(a.pairs[:P], b.pairs[:P])
        assert torch.equal(a.aabb.view(torch.int32), b.aabb.view(torch.int32))
        for k in ("norm", "cpta", "cptb", "depth", "bids"):
            assert torch.equal(getattr(a, k)[:C].view(torch.int32), getattr(b, k)[:C].view(torch.int32)), k
        seen.append(P)
    assert max(seen) > 0
