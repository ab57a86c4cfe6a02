"""Unrotated and axis-turned bodies in the exact MPR: portal normals and support
directions along axes (components that are zero of either sign), directions along a
cylinder's axis, and unit vectors one unit below length 1 all stay on its fast
path. Contacts equal the FP64 oracle's to float rounding, in every type pairing."""
import numpy as np
import pytest

import oracle as O
from _helpers import contact_errors
from collide_b200 import scenes as S
from test_gpu_narrowphase import check_exact, run_np, scale_of

pytestmark = pytest.mark.gpu

TURNS = {"none": [1, 0, 0, 0], "negative": [-1, 0, 0, 0], "half x": [0, 1, 0, 0], "half z": [0, 0, 0, 1],
         "quarter y": [0.5 ** 0.5, 0, 0.5 ** 0.5, 0]}


@pytest.mark.parametrize("jitter", [0.0, 0.002])
@pytest.mark.parametrize("turn", list(TURNS))
def test_lattice(cb, turn, jitter):
    rng = np.random.Generator(np.random.PCG64(4))
    c = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3) - 4.0
    n = len(c)
    T = rng.choice([S.SPHERE, S.ELLIPSOID, S.BOX, S.CYLINDER], size=n).astype(np.int32)
    B = np.full((n, 3), 0.505)
    B[T == S.SPHERE, 1:] = 0.0
    m = S._one_shape_per_body(T, B, c + jitter * rng.standard_normal((n, 3)), np.tile(TURNS[turn], (n, 1)), "lattice")
    m.pos[m.pos == 0.0] = -0.0
    _, p = O.broadphase(O.aabb(m), (9, 9, 9))
    ref = O.narrowphase(m, p, 0.0, "f64")
    got = run_np(cb, m, p)
    assert got["n"] == ref["n"] > 1500
    assert len({tuple(t) for t in T[np.stack([p >> 32, p & 0xFFFFFFFF], 1)][:].tolist()}) == 16
    check_exact(contact_errors(got, ref, scale_of(m)))
