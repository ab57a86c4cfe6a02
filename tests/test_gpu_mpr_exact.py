"""The exact MPR kernel at the counts where its lanes are dealt out differently
(a pair is two lanes, a warp at most sixteen pairs, two to six blocks of two
warps per SM, then a queue) and on directions with zero components (unrotated
boxes and cylinders), which leave its fast normalizations: contacts equal the
FP64 oracle's to float rounding."""
import numpy as np
import pytest

import oracle as O
from _helpers import contact_errors
from collide_b200 import scenes as S
from test_gpu_narrowphase import check_exact, run_np, scale_of

pytestmark = pytest.mark.gpu

SM = 148


@pytest.fixture(scope="module")
def heap():
    m = S.mixed_slab(16000, seed=5, extent=(0.24, 0.24, 0.12))
    _, p = O.broadphase(O.aabb(m), (20, 20, 10))
    assert len(p) > 6 * SM * 2 * 16 + 33
    return m, p


@pytest.mark.parametrize("count", [1, 2, 15, 16, 17, 31, 33, 4 * SM - 1, 4 * SM, 4 * SM + 1, 64 * SM - 1, 64 * SM + 1,
                                   6 * SM * 32 - 1, 6 * SM * 32, 6 * SM * 32 + 33])
def test_pair_counts(cb, heap, count):
    m, p = heap
    first = int(np.nonzero(m.T[p >> 32] != m.T[p & 0xFFFFFFFF])[0][0])  # a pair that is not sphere-sphere
    q = p[first:first + 1] if count == 1 else p[:count]
    ref = O.narrowphase(m, q, 0.0, "f64")
    got = run_np(cb, m, q)
    assert got["n"] == ref["n"]
    if ref["n"]:
        check_exact(contact_errors(got, ref, scale_of(m)))


@pytest.mark.parametrize("turn", ["none", "quarter"])
def test_directions_with_zero_components(cb, turn):
    rng = np.random.Generator(np.random.PCG64(11))
    n = 600
    cell = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    T = rng.choice([S.SPHERE, S.ELLIPSOID, S.BOX, S.CYLINDER], size=n).astype(np.int32)
    B = np.full((n, 3), 0.55)
    B[T == S.SPHERE, 1:] = 0.0
    q = np.zeros((n, 4))
    q[:, 0] = 1.0
    if turn == "quarter":
        q[:] = [np.sqrt(0.5), 0.0, 0.0, np.sqrt(0.5)]
    m = S._one_shape_per_body(T, B, cell.astype(float), q, "lattice")
    _, p = O.broadphase(O.aabb(m), (10, 10, 10))
    ref = O.narrowphase(m, p, 0.0, "f64")
    got = run_np(cb, m, p)
    assert got["n"] == ref["n"] > 500
    check_exact(contact_errors(got, ref, scale_of(m)))
