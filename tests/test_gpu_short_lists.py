"""Short pair lists, ordered by counting behind the MPR, equal the in-order path
bit for bit: at the edges of warps, blocks and shared memory, in every precision,
and when the next call's list is far longer or shorter than the kernel was
launched for."""
import pytest
import torch

from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def pair_of_pipes(cb, scene, precision, cap):
    ctxs = [cb.Context(), cb.Context()]
    ctxs[0].set_narrowphase_overlap(False)
    for c in ctxs:
        c.set_narrowphase_precision(precision)
    return [cb.DevicePipeline(cb.DeviceScene(scene), ctx=c, pairs_cap=cap) for c in ctxs]


def same(a, b):
    P, C = a.run()
    assert b.run() == (P, C)
    assert torch.equal(a.pairs[:P], b.pairs[:P])
    for k in ("norm", "cpta", "cptb", "depth", "bids"):
        assert torch.equal(getattr(a, k)[:C].view(torch.int32), getattr(b, k)[:C].view(torch.int32)), k
    return P, C


@pytest.mark.parametrize("precision", ["exact", "fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 40, 700, 3000, 9000])
def test_equal_to_in_order(cb, n, precision):
    # 0 to about 4,000 pairs
    z = (n * 6e-6 / 4) ** (1 / 3)
    a, b = pair_of_pipes(cb, S.mixed_slab(n, seed=n, extent=(2 * z, 2 * z, z)), precision, 4 * n + 16)
    for _ in range(4):  # first sizes, stream launches, capture, replay
        P, _ = same(a, b)
    assert P <= 4096


@pytest.mark.parametrize("precision", ["exact", "fp64"])
def test_lists_that_grow_and_shrink(cb, precision):
    n = 20_000
    a, b = pair_of_pipes(cb, S.mixed_slab(n, seed=7, extent=(1.0, 1.0, 0.5)), precision, 40 * n)
    start = a.ds.pos.clone()
    seen = []
    for f in (1.0, 1.0, 1.0, 0.5, 0.5, 0.3, 1.0, 0.3, 0.4, 0.45, 0.5, 2.0, 0.25, 1.0):
        for p in (a, b):
            p.ds.pos.copy_(start * f)
        seen.append(same(a, b)[0])
    assert min(seen) < 500 and max(seen) > 8192, seen
