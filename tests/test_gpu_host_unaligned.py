"""Pinned host arrays at any byte address (packed into one buffer by the caller; R and
rot aligned to 16 bytes, as the header asks) give what aligned pageable ones give."""
import pytest
import torch

from collide_b200 import scenes as S
from test_gpu_host_moves import scene

pytestmark = pytest.mark.gpu


def off_by_bytes(t, k):
    raw = t.contiguous().view(torch.uint8).reshape(-1)
    buf = torch.empty(raw.numel() + 16, dtype=torch.uint8).pin_memory()
    buf[k:k + raw.numel()].copy_(raw)
    return buf[k:k + raw.numel()]


@pytest.mark.parametrize("first", [1, 2, 3])
@pytest.mark.parametrize("only", [None, 0, 3])  # every array but R and rot, the types alone, C alone
@pytest.mark.parametrize("n", [3, 1000, 30_011])
def test_equal_to_copies(cb, n, only, first):
    m = scene(n)
    assert (m.T == S.CONE).any()  # C is read
    a = cb.HostSession(m, ctx=cb.Context(), pinned=False, pairs_cap=8 * n + 16)
    b = cb.HostSession(m, ctx=cb.Context(), pairs_cap=8 * n + 16)
    b.inputs = [off_by_bytes(t, first) if (k == only if only is not None else k not in (4, 7)) else t
                for k, t in enumerate(b.inputs)]
    for _ in range(2):
        P, C = a.run()
        assert b.run() == (P, C)
        assert torch.equal(a.pairs[:P], b.pairs[:P])
        for k in ("norm", "cpta", "cptb", "depth", "bids"):
            assert torch.equal(getattr(a, k)[:C].view(torch.int32), getattr(b, k)[:C].view(torch.int32)), k
