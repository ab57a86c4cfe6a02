"""Cells of many entries (ordered by body, tested by masks, written row by row
and merged) through every entry point that can meet them, and at the sizes where
their kernels change: 256-row items and column tiles, 4,096 entries (one block's
sort), buckets of 1,024 and 8,192 keys (merged by a warp, by a block). Pairs
equal the oracle's."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from _helpers import contact_errors, same_bits
from collide_b200 import scenes as S
from test_gpu_narrowphase import check_exact

pytestmark = pytest.mark.gpu


def dense_scene(n, seed=2):
    return S.clustered_spheres(n, seed=seed, clusters=2, sigma=0.01, background=0.05)


@pytest.mark.parametrize("k", [129, 255, 256, 257, 511, 513, 1025, 2049, 4095, 4097, 9000])
def test_one_crowded_cell(cb, k):
    # k boxes around one point (every pair of them overlaps or nearly so) among sparse ones
    rng = np.random.Generator(np.random.PCG64(k))
    n = k + 3000
    c = rng.random((n, 3)).astype(np.float32)
    c[rng.permutation(n)[:k]] = (0.5 + 0.004 * rng.standard_normal((k, 3))).astype(np.float32)
    r = np.float32(0.0025)
    a = np.concatenate([c - r, c + r])
    sh, p = O.broadphase(a, (30, 30, 30))
    ctx = cb.Context()
    for _ in range(3):  # found out by the chains, tested twice, masks kept
        t = torch.from_numpy(a.copy()).cuda()
        got = cb.Broadphase(ctx).detectPossibleCollisions(t)
        assert np.array_equal(got.cpu().numpy(), p)
        assert same_bits(t.cpu().numpy(), sh)


@pytest.mark.parametrize("overlap", [True, False])
def test_collide_on_a_crowded_scene(cb, overlap):
    sc = dense_scene(20_000)
    _, p = O.broadphase(O.aabb(sc), (64, 64, 64))
    ref = O.narrowphase(sc, p, 0.0, "f64")
    ctx = cb.Context()
    ctx.set_narrowphase_overlap(overlap)
    pipe = cb.DevicePipeline(cb.DeviceScene(sc), ctx=ctx, pairs_cap=len(p) + 10)
    for _ in range(4):  # chains, stream launches, capture, replay
        assert pipe.run() == (len(p), ref["n"])
        k = pipe.n_contacts
        keys = pipe.pairs[: len(p)].cpu().numpy()
        assert np.array_equal(np.sort(keys), p) and np.array_equal(keys[:k], ref["pairs"][:k])
        got = dict(contact_pairs=keys[:k], norm=pipe.norm[:k].cpu().numpy(), cpta=pipe.cpta[:k].cpu().numpy(),
                   cptb=pipe.cptb[:k].cpu().numpy(), depth=pipe.depth[:k].cpu().numpy())
        check_exact(contact_errors(got, ref, float(sc.B.max())))


def test_batch_with_a_crowded_scene(cb):
    from collide_b200 import _lib
    scenes = [S.mixed_slab(3000, seed=1, extent=(0.3, 0.3, 0.1)), dense_scene(8000), S.spheres_uniform(2000, seed=3)]
    per = [O.broadphase(O.aabb(s), (32, 32, 32))[1] for s in scenes]
    first = np.cumsum([0] + [s.n for s in scenes[:-1]])
    want = np.concatenate([p + (np.int64(f) << 32) + f for p, f in zip(per, first)])
    db = cb.DeviceBatch(scenes)
    bp = cb.BatchPipeline(db, ctx=cb.Context(), pairs_cap=16)
    counts = np.zeros(3, np.uint64)
    for _ in range(2):
        st = _lib.lib.cc_collide_batch(bp.ctx.h, ctypes.byref(bp.batch), 16, 16, 16, 0.0, ctypes.byref(bp.res),
                                       counts.ctypes.data, None, ctypes.c_void_p(0))
        assert st == _lib.CC_ERR_CAPACITY and counts.tolist() == [len(p) for p in per]
    for _ in range(4):
        n, k = bp.run()
        assert n == len(want) and np.array_equal(np.sort(bp.pairs[:n].cpu().numpy()), want)
        assert bp.scene_pairs.tolist() == [len(p) for p in per] and bp.contact_offsets[-1] == k


def test_incremental_and_host_steps_on_a_crowded_scene(cb):
    sc = dense_scene(12_000, seed=7)
    _, p = O.broadphase(O.aabb(sc), (64, 64, 64))
    ctx = cb.Context()
    ctx.set_incremental(True, 0.5)
    pipe = cb.DevicePipeline(cb.DeviceScene(sc), ctx=ctx, pairs_cap=len(p) + 10)
    for _ in range(3):
        pipe.run()
        assert np.array_equal(np.sort(pipe.pairs[: pipe.n_pairs].cpu().numpy()), p)
    hs = cb.HostSession(sc, ctx=cb.Context(), pairs_cap=len(p) + 10)
    for _ in range(3):
        hs.submit()
        hs.submit()
        for _ in range(2):
            hs.wait()
            assert np.array_equal(np.sort(hs.pairs[: hs.n_pairs].numpy()), p)
