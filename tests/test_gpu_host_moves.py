"""Host arrays moved by kernel (pinned, mapped memory) give what the copies give
(pageable memory): odd sizes, shapes whose C is read, boxes asked for, arrays that
start off a 16-byte boundary, and outputs that were too small."""
import numpy as np
import pytest
import torch

from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def scene(n):
    z = (n * 6e-6 / 4) ** (1 / 3)
    m = S.mixed_slab(n, seed=n, extent=(2 * z, 2 * z, z))
    cones = np.arange(0, n, 7)
    m.T[cones] = S.CONE
    m.C[cones] = np.random.Generator(np.random.PCG64(n)).uniform(0.001, 0.004, (len(cones), 3))
    return m


def off_by(t, words):
    """The same contents, pinned, `words` elements behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + words, dtype=t.dtype).pin_memory()
    buf[words:].copy_(t.reshape(-1))
    return buf[words:].view(t.shape)


@pytest.mark.parametrize("boxes", [False, True])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 17, 1000, 4097, 30_011])
def test_equal_to_copies(cb, n, shift, boxes):
    m = scene(n)
    a = cb.HostSession(m, ctx=cb.Context(), want_aabb=boxes, pinned=False, pairs_cap=8 * n + 16)
    b = cb.HostSession(m, ctx=cb.Context(), want_aabb=boxes, pairs_cap=8 * n + 16)
    if shift:  # R and rot (real4) have to stay aligned
        b.inputs = [t if k in (4, 7) else off_by(t, shift) for k, t in enumerate(b.inputs)]
    for _ in range(4):
        P, C = a.run()
        assert b.run() == (P, C)
        assert torch.equal(a.pairs[:P], b.pairs[:P])
        for k in ("norm", "cpta", "cptb", "depth", "bids"):
            assert torch.equal(getattr(a, k)[:C].view(torch.int32), getattr(b, k)[:C].view(torch.int32)), k
        if boxes:
            assert torch.equal(a.aabb.view(torch.int32), b.aabb.view(torch.int32))
        for x in (a, b):  # other poses next time
            x.inputs[6].mul_(0.97)


def test_outputs_too_small_then_grown(cb):
    m = scene(5000)
    a = cb.HostSession(m, ctx=cb.Context(), pinned=False, pairs_cap=60_000)
    b = cb.HostSession(m, ctx=cb.Context(), pairs_cap=100)
    P, C = a.run()
    assert P > 100 and b.run() == (P, C)
    assert torch.equal(a.pairs[:P], b.pairs[:P]) and torch.equal(a.norm[:C], b.norm[:C])
