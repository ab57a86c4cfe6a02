"""Calls with little free memory. Chained cells and the dense-cell test need more
scratch than a plain search on sorted cells: where it is refused the call runs on
the latter, and later calls with room give the same list."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from collide_b200 import _lib
from collide_b200 import scenes as S

pytestmark = pytest.mark.gpu

N = 2_000_000


@pytest.fixture(scope="module")
def scene():
    sc = S.spheres_uniform(N, seed=3, rmin=0.0005, rmax=0.002)
    a = S.sphere_aabbs(sc)
    return a, O.broadphase(a, (64, 64, 64))[1]


# the plain search gets by with 260 MB; chained cells take 340, the dense cells' copies 280 more
@pytest.mark.parametrize("grid,mb", [((0, 0, 0), 300), ((12, 12, 12), 470), ((12, 12, 12), 300), ((12, 12, 12), 340)])
def test_broadphase(cb, scene, grid, mb):
    a, p = scene
    boxes = torch.from_numpy(a).cuda()
    out, n_pairs = torch.zeros(len(p) + 100, dtype=torch.int64, device="cuda"), ctypes.c_uint64()
    warm = cb.Context()  # loads the kernels
    warm.set_search_grid(grid)

    def call(ctx):
        t = boxes.clone()
        st = _lib.lib.cc_broadphase(ctx.h, N, t.data_ptr(), 16, 16, 16, out.data_ptr(), out.numel(), ctypes.byref(n_pairs),
                                    None)
        ctx.check(st, "cc_broadphase")
        assert n_pairs.value == len(p) and np.array_equal(out[: len(p)].cpu().numpy(), p)

    call(warm)
    del warm
    ctx = cb.Context()
    ctx.set_search_grid(grid)
    held = torch.empty(torch.cuda.mem_get_info()[0] - (mb << 20), dtype=torch.uint8, device="cuda")
    for _ in range(3):
        call(ctx)
    del held
    torch.cuda.empty_cache()
    for _ in range(36):  # chained cells are tried again
        call(ctx)
