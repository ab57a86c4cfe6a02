"""Incremental steps over a floor: the first rebuild finds out that a body lies in many
search cells, the later ones go straight to sorted cells. Results equal full steps'."""
import numpy as np
import pytest
import torch

from collide_b200 import scenes as S
from test_gpu_floor import on_floor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,width", [(5_000, 1.6), (40_000, 4.5)])
def test_rebuilds(cb, n, width):
    sc, flat = on_floor(n, 3, width), S.mixed_slab(n, seed=3, extent=(width, width, 0.012))
    a, b, f = cb.DeviceScene(sc), cb.DeviceScene(sc), cb.DeviceScene(flat)
    ctx, plain = cb.Context(), cb.Context()
    for c in (ctx, plain):
        c.set_incremental(True, 0.5)
    x = cb.DevicePipeline(a, ctx=ctx, pairs_cap=8 * n)
    y = cb.DevicePipeline(b, ctx=cb.Context(), pairs_cap=8 * n)
    z = cb.DevicePipeline(f, ctx=plain, pairs_cap=8 * n)
    rng, launches = np.random.Generator(np.random.PCG64(1)), []
    for _ in range(6):  # every step moves too far for the list
        d = torch.from_numpy((0.01 * rng.standard_normal((n, 3))).astype(np.float32)).cuda()
        for s in (a, b, f):
            s.pos[:n] += d
        P, C = y.run()
        z.run()
        assert x.run() == (P, C) and C > 0
        assert torch.equal(x.pairs[:P], y.pairs[:P]) and torch.equal(x.norm[:C], y.norm[:C])
        assert ctx.last_step_rebuilt() and plain.last_step_rebuilt()
        launches.append(ctx.launches() - plain.launches())
    # sorted cells take two launches more than chained ones; both one after the other took ten
    assert max(launches[1:]) <= 4, launches
