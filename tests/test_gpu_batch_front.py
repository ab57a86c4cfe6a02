"""The batch pass's first and last kernels where they can go wrong: more scenes
than a block has threads, scenes of zero to three hundred shapes across tile
edges, cones (whose third array the gather has to copy), the same scenes
gathered from their own allocations, and the pair counts of an output that is
too small. Boxes and pairs equal the oracle's per scene, bit for bit."""
import ctypes

import numpy as np
import pytest

import oracle as O
from _helpers import same_bits
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu


def uneven_scenes(count, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i in range(count):
        n = int(rng.choice([0, 1, 2, 7, 64, 255, 256, 300], p=[0.1, 0.2, 0.2, 0.2, 0.1, 0.05, 0.05, 0.1]))
        sc = S.mixed_slab(n, seed=seed * 7919 + i, extent=(0.05, 0.05, 0.03))
        cone = rng.random(n) < 0.1  # bounded as a triangle of A, B, C
        sc.T[cone] = S.CONE
        for f in (sc.A, sc.B, sc.C):
            f[cone] = rng.uniform(0.001, 0.006, size=(int(cone.sum()), 3))
        out.append(sc)
    return out


def oracle_of(scenes):
    box, pairs, first = [], [], 0
    for sc in scenes:
        if sc.n:
            sh, p = O.broadphase(O.aabb(sc), (16, 16, 16))
            box.append(sh)
            pairs.append(p + (np.int64(first) << 32) + first)
            first += sc.n
    lo = np.concatenate([b[:len(b) // 2] for b in box])
    hi = np.concatenate([b[len(b) // 2:] for b in box])
    return np.concatenate([lo, hi]), np.concatenate(pairs)


@pytest.mark.parametrize("count", [1, 3, 255, 256, 257, 700])
def test_uneven_scenes_batched_and_gathered(cb, count):
    scenes = uneven_scenes(count, seed=count) + [S.mixed_slab(300, seed=1, extent=(0.05, 0.05, 0.03))]
    box, pairs = oracle_of(scenes)
    db = cb.DeviceBatch(scenes)
    bp = cb.BatchPipeline(db, ctx=cb.Context())
    sp = cb.ScenesPipeline(cb.Context())
    held = [cb.DeviceScene(s) for s in scenes]
    per = np.zeros(len(scenes), np.int64)
    np.add.at(per, np.searchsorted(db.shape_offsets.astype(np.int64), pairs >> 32, side="right") - 1, 1)
    for _ in range(3):  # stream launches, capture, replay
        results = []
        for p, got in ((bp, bp.run()), (sp, sp.run(held))):
            assert got[0] == len(pairs)
            assert same_bits(p.aabb[: 2 * db.n].cpu().numpy(), box)
            keys = p.pairs[: got[0]].cpu().numpy()
            assert np.array_equal(np.sort(keys), pairs)
            assert np.array_equal(p.scene_pairs.astype(np.int64), per)
            off = p.contact_offsets.astype(np.int64)
            assert off[0] == 0 and off[-1] == got[1] and np.all(np.diff(off) >= 0)
            hit = keys[: got[1]] >> 32
            assert np.array_equal(off, np.searchsorted(hit, db.shape_offsets.astype(np.int64)))
            results.append((keys, p.norm[: got[1]].cpu().numpy(), p.depth[: got[1]].cpu().numpy()))
        for a, b in zip(*results):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_pair_counts_of_an_output_too_small(cb):
    from collide_b200 import _lib
    scenes = uneven_scenes(40, seed=3)
    _, pairs = oracle_of(scenes)
    db = cb.DeviceBatch(scenes)
    bp = cb.BatchPipeline(db, ctx=cb.Context(), pairs_cap=8)
    assert len(pairs) > 8
    counts = np.zeros(db.num_scenes, np.uint64)
    for _ in range(2):
        st = _lib.lib.cc_collide_batch(bp.ctx.h, ctypes.byref(bp.batch), 16, 16, 16, 0.0, ctypes.byref(bp.res),
                                       counts.ctypes.data, None, ctypes.c_void_p(0))
        assert st == _lib.CC_ERR_CAPACITY and bp.res.n_pairs == len(pairs)
        so = db.shape_offsets.astype(np.int64)
        want = np.searchsorted(pairs >> 32, so[1:]) - np.searchsorted(pairs >> 32, so[:-1])
        assert np.array_equal(counts.astype(np.int64), want)
