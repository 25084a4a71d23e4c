"""What a context does around the line kernel: which calls run on it, and what
becomes of them without it."""
import numpy as np
import pytest

import oracle as O
import plastimatch_b200 as P
from conftest import rel_err
from plastimatch_b200 import synth
from plastimatch_b200.geometry import BsplineGrid

pytestmark = pytest.mark.gpu


def _case(dim=(48, 40, 36), vpr=(5, 6, 4), seed=31):
    fixed = synth.gaussian_blobs(dim, spacing=(1.0, 1.1, 1.6), seed=seed)
    g0 = BsplineGrid.for_volume(fixed, 8)
    moving = synth.warp_trilinear(fixed, fixed, g0,
                                  synth.random_coeff(g0, 1.5, seed + 1))
    grid = BsplineGrid.for_volume(fixed, vpr)
    return fixed, moving, grid, synth.random_coeff(grid, 1.0, seed + 2)


def test_without_room_for_its_buffers_a_context_keeps_the_tile_kernel():
    """The last request of a creation is the line kernel's buffers.  Without
    them the context evaluates on the tile kernel, with the same results as
    one that is pinned to it; every earlier failure is a failed creation."""
    fixed, moving, grid, coeff = _case()
    lib = P.lib()
    nth = 0
    while True:
        nth += 1
        assert nth < 40
        lib.b200bsp_debug_fail_alloc(nth)
        try:
            ctx = P.Context(fixed, moving, grid)
        except P.B200Error as e:
            assert "injected" in str(e)
            continue
        finally:
            lib.b200bsp_debug_fail_alloc(0)
        break
    with ctx, P.Context(fixed, moving, grid, tc_kernel="tile") as tile:
        for c in (ctx, tile):
            c.set_images()
        assert ctx.mse_kernel()[0] == "tile"
        for call in ("score_mse", "score_mi"):
            got, want = getattr(ctx, call)(coeff), getattr(tile, call)(coeff)
            assert got[0] == want[0] and got[2] == want[2] > 0
            np.testing.assert_array_equal(got[1], want[1])
