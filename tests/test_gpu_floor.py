"""Scenes whose contacts share one body, a floor behind or before all others: most
contacts then start at a few slots of the contact hash, which overflows, and the
narrowphase is redone in order. Pairs, contacts and a batch's offsets equal those
of the path that sorts first, call after call."""
import numpy as np
import pytest
import torch

from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def on_floor(n, seed, width, last=True):
    """A thin layer of n bodies, about half of them touching a box of the layer's area."""
    m = S.mixed_slab(n, seed=seed, extent=(width, width, 0.012))
    f = S._one_shape_per_body(np.array([S.BOX]), np.array([[width / 2, width / 2, 0.02]]),
                              np.array([[width / 2, width / 2, -0.017]]), S._identity_quats(1), "floor")
    a, b = (m, f) if last else (f, m)
    k = {x: np.concatenate([getattr(a, x), getattr(b, x)]) for x in ("T", "A", "B", "C", "R", "pos", "rot", "active")}
    return S.Scene(ID=np.arange(n + 1, dtype=np.uint32), **k)


def equal_to_in_order(a, b, calls=4):
    a.ctx.set_narrowphase_overlap(False)
    for call in range(calls):
        P, C = a.run()
        assert b.run() == (P, C) and C > 0
        assert torch.equal(a.pairs[:P], b.pairs[:P]), call
        for k in ("norm", "cpta", "cptb", "depth", "bids"):
            assert torch.equal(getattr(a, k)[:C].view(torch.int32), getattr(b, k)[:C].view(torch.int32)), (call, k)
        keys = b.pairs.cpu().numpy()
        assert (np.diff(keys[:C]) > 0).all() and (np.diff(keys[C:P]) > 0).all()
    return P, C


@pytest.mark.parametrize("last", [True, False])
@pytest.mark.parametrize("n,width", [(8_000, 2.0), (20_000, 3.0)])
def test_one_scene(cb, n, width, last):
    sc = on_floor(n, 5, width, last)
    a, b = (cb.DevicePipeline(cb.DeviceScene(sc), ctx=cb.Context(), pairs_cap=4 * n) for _ in range(2))
    P, C = equal_to_in_order(a, b)
    floor = n if last else 0
    assert P > 4096 and int((b.bids[:C] == floor).any(1).sum()) > 3000


def test_batch(cb):
    scenes = [on_floor(k, k, w) for k, w in ((9_000, 2.0), (700, 0.6), (12_000, 2.5))]
    db = cb.DeviceBatch(scenes)
    a, b = (cb.BatchPipeline(db, ctx=cb.Context(), pairs_cap=4 * db.n) for _ in range(2))
    for _ in range(3):
        P, C = equal_to_in_order(a, b, 1)
        first = np.searchsorted(b.pairs[:C].cpu().numpy(), db.shape_offsets.astype(np.int64) << 32)
        assert np.array_equal(b.contact_offsets.astype(np.int64), first)
        owner = b.pairs[:P].cpu().numpy() >> 32
        want = np.histogram(owner, bins=db.shape_offsets.astype(np.int64))[0]
        assert np.array_equal(b.scene_pairs.astype(np.int64), want)


def test_no_redo_where_contacts_share_a_body(cb):
    # the same scene with the floor first and last: as many launches a step (a redo takes two more)
    n, launches = 7_500, []
    for last in (False, True):
        sc = on_floor(n, 5, 2.0, last)
        pipe = cb.DevicePipeline(cb.DeviceScene(sc), ctx=cb.Context(), pairs_cap=4 * n)
        for _ in range(4):
            P, C = pipe.run()
        floor = n if last else 0
        assert P > 4096 and 3000 < int((pipe.bids[:C] == floor).any(1).sum()) < 4000
        launches.append(pipe.ctx.launches())
    assert launches[0] == launches[1]
