"""The line kernel (what a tensor-core-form context runs by default on grids
with 3 to 10 voxels a region) against the FP32 form's tile kernel, at the
edges of its blocks: warps and blocks partly beyond the ROI, ragged last
tiles, the smallest and largest regions, rotated axes, partial ROIs, images
wider than one finish block.

Both kernels work in float and differ in the order of their sums: the field
by a few units of 2^-24 of the coefficients, the gradient by the rounding of
sums of at most 4 x 4 x 4 tiles of 1000 voxels (grouped, < 100 roundings
deep), i.e. 100 x 2^-24 = 6e-6; a voxel whose position falls on the other
side of a cell's face changes its own term only (images without noise: the
moving gradient is smooth).  Bars: score 2e-6, gradient 2e-5, count 1e-4 + 2.
"""
import numpy as np
import pytest

import plastimatch_b200 as P
from conftest import rel_err
from plastimatch_b200 import synth
from plastimatch_b200.geometry import BsplineGrid, Volume

pytestmark = pytest.mark.gpu

# dims, vox_per_rgn, ROI (offset, dim) or None, rotation about z (degrees)
CASES = [
    ((24, 24, 24), (4, 4, 4), None, 0.0),
    ((33, 9, 7), (3, 3, 3), None, 0.0),            # one lane in the last warp
    ((65, 41, 30), (10, 3, 9), None, 8.0),
    ((129, 31, 17), (5, 10, 10), None, 0.0),       # two planes in the last row
    ((64, 64, 64), (3, 10, 10), None, 5.0),
    ((31, 200, 11), (7, 4, 3), None, 0.0),         # less than a warp along x
    ((70, 50, 40), (6, 5, 7), ((5, 3, 2), (57, 41, 31)), 0.0),
    ((1040, 20, 12), (10, 6, 4), None, 0.0),       # two finish blocks along x
    ((48, 44, 36), (8, 9, 6), ((1, 0, 3), (47, 44, 33)), -15.0),
]
# blocks whose dynamic shared memory lies just below 48 KB, where the static
# arrays beside it need the larger limit
LARGE_BLOCKS = [((224, 529, 28), (3, 3, 9), None, 0.0),
                ((81, 439, 106), (4, 3, 10), None, 0.0)]
# more blocks of the rows' contraction than the chip holds at once, of two
# and of one block an SM; one part a tile and eight
CONTRACTIONS = [((300, 590, 40), (10, 3, 4), None, 0.0),
                ((300, 590, 50), (10, 3, 5), None, 0.0),
                ((40, 44, 81), (4, 10, 9), None, 0.0)]


def _volume(dim, seed, dcos, origin=(0.0, 0.0, 0.0)):
    v = synth.gaussian_blobs(dim, spacing=(1.0, 1.1, 1.6), seed=seed,
                             noise_sigma=0.0)
    return Volume(v.img, origin=origin, spacing=v.spacing, dcos=dcos)


def _case(dim, vpr, roi, angle, seed=71):
    a = np.deg2rad(angle)
    dcos = (np.cos(a), -np.sin(a), 0.0, np.sin(a), np.cos(a), 0.0, 0.0, 0.0, 1.0)
    fixed = _volume(dim, seed, dcos)
    # another extent and place: some voxels land outside on every axis
    moving = _volume((dim[0] - 2, dim[1] + 3, dim[2] + 1), seed, dcos,
                     (0.4, -0.7, 0.3))
    kw = dict(roi_offset=roi[0], roi_dim=roi[1]) if roi else {}
    grid = BsplineGrid.for_volume(fixed, vpr, **kw)
    return fixed, moving, grid, synth.random_coeff(grid, 1.5, seed + 2)


@pytest.mark.parametrize("grad", ["nearest", "trilinear"])
@pytest.mark.parametrize("case", CASES + LARGE_BLOCKS + CONTRACTIONS)
def test_line_kernel_matches_tile_kernel(case, grad):
    fixed, moving, grid, coeff = _case(*case)
    out = []
    for form in ("fp32", "tc"):
        with P.Context(fixed, moving, grid, form=form, mse_grad=grad) as ctx:
            ctx.set_images()
            name = ctx.mse_kernel()[0]
            assert name == ("fp32" if form == "fp32" else "line")
            out.append(ctx.score_mse(coeff))
            again = ctx.score_mse(coeff)
            assert again[0] == out[-1][0] and again[2] == out[-1][2]
            np.testing.assert_array_equal(again[1], out[-1][1])
    (s0, g0, n0), (s1, g1, n1) = out
    assert n0 > 0 and abs(n1 - n0) <= 1e-4 * n0 + 2, (n1, n0)
    assert abs(s1 - s0) <= 2e-6 * abs(s0), (s1, s0)
    assert rel_err(g1, g0) < 2e-5, rel_err(g1, g0)


def test_regions_outside_the_line_kernel_keep_the_tile_kernel():
    f = _volume((40, 48, 24), 3, (1, 0, 0, 0, 1, 0, 0, 0, 1))
    for vpr in ((5, 12, 5), (2, 5, 5), (5, 5, 11)):
        with P.Context(f, f, BsplineGrid.for_volume(f, vpr)) as ctx:
            assert ctx.mse_kernel()[0] == "tile"


@pytest.mark.parametrize("window,bins", [("pvi8", 20), ("pvi8", 64),
                                         ("parzen", 32), ("parzen", 5)])
@pytest.mark.parametrize("case", [c for c in CASES if c[2] is None])
def test_line_kernel_mi_matches_tile_kernel(case, window, bins):
    """Mattes MI: the line kernel's histograms (and, for Parzen windows, its
    gradient) against the FP32 form's.  The weights are sums of 2^-24 units of
    positions that agree to some 2^-21 voxel, so the histograms agree to 1e-6
    of their counts times the few voxels per bin edge: bar 1e-5; the score, a
    sum over them, 1e-5; the Parzen gradient, whose window derivative scales
    the same differences by at most 2 bins, 5e-5."""
    fixed, moving, grid, coeff = _case(*case)
    out = []
    for form in ("fp32", "tc"):
        with P.Context(fixed, moving, grid, form=form, mi_window=window,
                       mi_bins=bins) as ctx:
            ctx.set_images()
            out.append(ctx.score_mi(coeff, with_hist=True))
            h = ctx.mi_hist(coeff)
            np.testing.assert_array_equal(h, ctx.mi_hist(coeff))
            assert h[-1] == out[-1][2]
            if window == "pvi8":       # every voxel once, eight weights each
                assert h[:bins].sum() == h[-1]
                assert h[bins:2 * bins].sum() == h[2 * bins:-1].sum()
    (s0, g0, n0, h0), (s1, g1, n1, h1) = out
    assert n0 > 0 and abs(n1 - n0) <= 1e-4 * n0 + 2, (n1, n0)
    for a, b in zip(h1, h0):
        assert rel_err(a, b) < 1e-5 + 2.0 / n0, rel_err(a, b)
    assert abs(s1 - s0) <= 1e-5 * abs(s0) + 1e-6, (s1, s0)
    if window == "parzen":
        assert rel_err(g1, g0) < 5e-5, rel_err(g1, g0)


@pytest.mark.parametrize("case", CASES)
def test_line_kernel_field_and_warp(case):
    """The dense field against its double-precision evaluation (64 products
    of coefficients up to some 6 mm: 1e-5 mm), and the warp against the
    trilinear sample at those positions (1e-3 of the image's 1000 grey levels
    times a position error of 1e-4 voxel, away from the image's edge)."""
    fixed, moving, grid, coeff = _case(*case)
    off, dim = grid.roi_offset, grid.roi_dim
    roi = tuple(slice(off[d], off[d] + dim[d]) for d in (2, 1, 0))
    ref = synth.bspline_field(grid, coeff)
    for form in ("fp32", "tc"):
        with P.Context(fixed, moving, grid, form=form) as ctx:
            ctx.set_images()
            vf = ctx.interpolate_vf(coeff)
            np.testing.assert_allclose(vf[roi], ref, atol=1e-5)
            mask = np.ones(vf.shape[:3], bool)
            mask[roi] = False
            assert not vf[mask].any()
            if case[2] is not None:
                continue
            w = ctx.warp(coeff, -7.0)
    if case[2] is None:
        want = synth.warp_trilinear(moving, fixed, grid, coeff, -7.0).img
        bad = np.abs(w - want) > 0.1
        assert bad.mean() < 1e-4, bad.mean()


# below one part of the staged copies (65536 floats), three parts, four
# longer ones
@pytest.mark.parametrize("metric", ["mse", "mi"])
@pytest.mark.parametrize("dim", [(20, 18, 16), (90, 81, 78), (129, 129, 126)])
def test_score_with_host_outputs_is_the_device_one(dim, metric):
    """Host coefficients and outputs go through page-locked staging buffers
    around the same kernels: every bit of the results is the same, also when
    the host arrays are page-locked themselves."""
    import ctypes as C

    import torch
    fixed, moving, grid, coeff = _case(dim, (3, 3, 3), None, 0.0)
    reg = P.reg_parms(curvature=0.1, total_displacement=0.01)
    with P.Context(fixed, moving, grid, mi_window="pvi8") as ctx:
        ctx.set_images()
        host = ctx.score(coeff, metric, 0.5, reg)
        pinned = ctx.score(torch.from_numpy(coeff).pin_memory(), metric, 0.5,
                           reg)
        dc = torch.from_numpy(coeff).cuda()
        g = torch.empty_like(dc)
        s = torch.empty(2, device="cuda")
        n = torch.empty(1, dtype=torch.int64, device="cuda")
        rc = P.lib().b200bsp_score(
            ctx._h, dc.data_ptr(), 0 if metric == "mse" else 1, C.c_float(0.5),
            C.byref(reg), s.data_ptr(), g.data_ptr(), s.data_ptr() + 4,
            n.data_ptr())
        assert rc == 0
        torch.cuda.synchronize()
    for got in (host, pinned):
        assert got[0] == s[0].item() and got[2] == s[1].item()
        assert got[3] == n.item() and got[3] > 0
        assert np.array_equal(got[1], g.cpu().numpy())
