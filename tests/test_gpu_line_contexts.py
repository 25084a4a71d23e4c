"""What a context does around the line kernel: which calls run on it, and what
becomes of them without it."""
import numpy as np
import pytest

import oracle as O
import plastimatch_b200 as P
from conftest import rel_err
from plastimatch_b200 import synth
from plastimatch_b200.geometry import BsplineGrid, Volume

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


@pytest.mark.parametrize("angle", [0.0, 10.0])
@pytest.mark.parametrize("what", ["nearest", "trilinear", "parzen"])
def test_voxels_outside_leave_no_nan(what, angle):
    """A NaN in the moving image's first plane, which only voxels outside the
    image read (at x = -0.6; the next ones, at 1.7 and beyond, read planes 1
    and up), changes no bit of the results."""
    a = np.deg2rad(angle)
    dcos = (np.cos(a), -np.sin(a), 0.0, np.sin(a), np.cos(a), 0.0, 0.0, 0.0, 1.0)
    f = synth.gaussian_blobs((16, 30, 20), spacing=(1, 1, 1), seed=5).img
    m = synth.gaussian_blobs((40, 30, 20), spacing=(1, 1, 1), seed=6).img
    fixed = Volume(f, origin=(0.0, 0.0, 0.0), spacing=(2.3, 1.0, 1.0), dcos=dcos)
    # the moving image begins 0.6 mm along x behind the fixed one's origin
    moving = Volume(m, origin=(0.6 * dcos[0], 0.6 * dcos[3], 0.0),
                    spacing=(1.0, 1.0, 1.0), dcos=dcos)
    grid = BsplineGrid.for_volume(fixed, (4, 5, 6))
    coeff = synth.random_coeff(grid, 0.02, 7)
    kw = (dict(mi_window="parzen") if what == "parzen" else dict(mse_grad=what))
    out = []
    with P.Context(fixed, moving, grid, **kw) as ctx:
        assert ctx.mse_kernel()[0] == "line"
        for border in (float(m.mean()), np.nan):
            img = m.copy()
            img[:, :, 0] = border
            ctx.set_images(None, img)
            out.append(ctx.score_mi(coeff) if what == "parzen"
                       else ctx.score_mse(coeff))
    (s0, g0, n0), (s1, g1, n1) = out
    assert 0 < n0 == n1 < f.size and s0 == s1
    np.testing.assert_array_equal(g0, g1)


@pytest.mark.parametrize("call", ["score_mi", "score"])
def test_page_locked_gradients_are_copied_once(call):
    """A page-locked output takes the device's copy directly: the call takes
    at most half as long again as the copy (and 40 us) more than the one that leaves the
    gradient on the device.  Through the staging buffer a host memcpy comes
    on top, which takes longer than the copy."""
    import ctypes as C
    import time

    import torch
    fixed, moving, grid, coeff = _case((240, 200, 160), (3, 3, 3))
    lib = P.lib()
    dc = torch.from_numpy(coeff).cuda()
    dg = torch.empty_like(dc)
    hg = torch.empty(coeff.size).pin_memory()
    s, n = C.c_float(), C.c_int64()

    def best(fn):
        t = []
        for _ in range(20):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            fn()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)

    with P.Context(fixed, moving, grid) as ctx:
        ctx.set_images()

        def run(g):
            if call == "score_mi":
                rc = lib.b200bsp_score_mi(ctx._h, dc.data_ptr(), C.addressof(s),
                                          g.data_ptr(), C.addressof(n), None,
                                          None, None)
            else:
                rc = lib.b200bsp_score(ctx._h, dc.data_ptr(), 1, C.c_float(1.0),
                                       None, C.addressof(s), g.data_ptr(), None,
                                       C.addressof(n))
            assert rc == 0
        t_dev, t_host = best(lambda: run(dg)), best(lambda: run(hg))
        np.testing.assert_array_equal(hg.numpy(), dg.cpu().numpy())
    t_copy = best(lambda: hg.copy_(dg, non_blocking=True))
    assert t_host - t_dev < 1.5 * t_copy + 40e-6, (t_dev, t_host, t_copy)


def _field_64_taps(grid, coeff):
    """The field as the plain kernel sums it: float weights ((z y) x), one
    fused multiply-add a knot, x fastest (double products are exact, so that
    each sum is rounded to float once, up to the rare double rounding)."""
    f4 = np.float32
    nx, ny, nz = grid.roi_dim
    lut = [O.port_basis_lut(v).reshape(v, 4).astype(f4) for v in grid.vox_per_rgn]
    c = coeff.reshape(grid.cdims[2], grid.cdims[1], grid.cdims[0], 3)
    at = [np.arange(n) // v for n, v in zip((nx, ny, nz), grid.vox_per_rgn)]
    w = [t[np.arange(n) % v] for t, n, v in zip(lut, (nx, ny, nz), grid.vox_per_rgn)]
    d = np.zeros((nz, ny, nx, 3), f4)
    for k in range(4):
        for j in range(4):
            b = w[1][:, j][None, :] * w[2][:, k][:, None]
            for i in range(4):
                a = w[0][:, i][None, None, :] * b[:, :, None]
                t = c[at[2] + k][:, at[1] + j][:, :, at[0] + i]
                d = (a[..., None].astype(np.float64) * t + d).astype(f4)
    return d


@pytest.mark.parametrize("dim,kw", [
    ((48, 40, 36), dict(form="fp32")), ((48, 40, 36), dict(tc_kernel="tile")),
    ((48, 40, 36), dict(tc_kernel="xlane")), ((34, 34, 34), dict())])
def test_field_of_a_pinned_context_keeps_its_kernel(dim, kw):
    """The field of an FP32 context, and of one with a pinned tensor-core
    kernel, on a grid that the line kernel takes, and of a small image: the
    plain kernel's 64 products a voxel, bit for bit (but for double
    roundings, 1e-4 of the values at most), and the warp that goes with
    it."""
    fixed, moving, grid, coeff = _case(dim)
    want = _field_64_taps(grid, coeff)
    with P.Context(fixed, moving, grid, **kw) as ctx:
        ctx.set_images()
        vf = ctx.interpolate_vf(coeff)
        w = ctx.warp(coeff, -7.0)
    assert (vf != want).mean() <= 1e-4, (vf != want).mean()
    ref = synth.warp_trilinear(moving, fixed, grid, coeff, -7.0).img
    assert (np.abs(w - ref) > 0.1).mean() < 1e-4


def _noise(dim, origin, seed):
    nx, ny, nz = dim
    g = np.random.default_rng(seed)
    return Volume(g.random((nz, ny, nx), np.float32), origin=origin,
                  spacing=(1.0, 1.0, 1.0))


@pytest.mark.parametrize("bins", [3, 20, 64])
@pytest.mark.parametrize("dim,vpr", [((70, 60, 50), (4, 5, 6)),
                                     ((512, 512, 64), (10, 10, 4))])
def test_histograms_of_noise(dim, vpr, bins):
    """Images whose neighbours share no bin: a voxel's eight weights fall into
    many.  Without a displacement both forms compute the same positions, so
    every integer of the histograms is the FP32 form's -- but where all eight
    weights of a voxel share a bin (3 bins: one voxel in 2187; none else) the
    line kernel adds their sum, 2^24, for eight roundings of half a unit."""
    fixed = _noise(dim, (0.0, 0.0, 0.0), 3)
    moving = _noise(dim, (-0.37, 0.41, -0.29), 4)
    grid = BsplineGrid.for_volume(fixed, vpr)
    h = []
    for form in ("fp32", "tc"):
        with P.Context(fixed, moving, grid, form=form, mi_bins=bins) as ctx:
            ctx.set_images()
            h.append(ctx.mi_hist(np.zeros(grid.num_coeff, np.float32)))
    assert h[0][-1] > 0.9 * fixed.img.size
    if bins == 3:
        assert np.abs(h[1][bins:] - h[0][bins:]).sum() <= 2 * 4 * fixed.img.size / 1000
        np.testing.assert_array_equal(h[1][:bins], h[0][:bins])
    else:
        np.testing.assert_array_equal(h[1], h[0])


@pytest.mark.parametrize("bins", [20, 64])
def test_histograms_of_noise_take_no_longer(bins):
    """The same images, timed: pass 1 on the line kernel against the tile
    kernel's (which took 0.1 to 0.2 times as long when the line kernel's
    weights for a third bin went to the histogram in memory)."""
    import time
    fixed = _noise((128, 128, 64), (0.0, 0.0, 0.0), 3)
    moving = _noise((128, 128, 64), (-0.37, 0.41, -0.29), 4)
    grid = BsplineGrid.for_volume(fixed, 5)
    coeff = synth.random_coeff(grid, 0.5, 5)
    t = []
    for kernel in ("tile", "auto"):
        with P.Context(fixed, moving, grid, mi_bins=bins,
                       tc_kernel=kernel) as ctx:
            ctx.set_images()
            best = np.inf
            for _ in range(20):
                t0 = time.perf_counter()
                ctx.mi_hist(coeff)
                best = min(best, time.perf_counter() - t0)
            t.append(best)
    assert t[1] < 1.1 * t[0], t


def _mi_device(ctx, coeff, out):
    """b200bsp_score (MI) with device outputs, stream-ordered."""
    import ctypes as C
    rc = P.lib().b200bsp_score(
        ctx._h, coeff.data_ptr(), 1, C.c_float(1.0), None, out[0].data_ptr(),
        out[1].data_ptr(), None, out[2].data_ptr())
    assert rc == 0


def test_new_images_reach_pass_1():
    """PVI-8's pass 1 reads an image of the moving bins that its first
    evaluation forms: after b200bsp_set_images it is the new one, in direct
    calls and in a graph captured before."""
    import torch
    fixed, moving, grid, coeff = _case()
    other = synth.gaussian_blobs(moving.dim, spacing=moving.spacing, seed=77)
    with P.Context(fixed, other, grid) as ctx:
        ctx.set_images()
        s_new, g_new, n_new = ctx.score_mi(coeff)
    dc = torch.from_numpy(coeff).cuda()

    def outputs():
        return (torch.zeros(1, device="cuda"), torch.zeros_like(dc),
                torch.zeros(1, dtype=torch.int64, device="cuda"))
    stream = torch.cuda.Stream()
    for evaluate_first in (False, True):
        with P.Context(fixed, moving, grid) as ctx:
            ctx.set_stream(stream.cuda_stream)
            ctx.set_images()
            if evaluate_first:
                s_old = ctx.score_mi(coeff)[0]
                assert s_old != s_new
            out, graph = outputs(), torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream,
                                  capture_error_mode="relaxed"):
                _mi_device(ctx, dc, out)
            ctx.set_images(None, other.img)
            graph.replay()
            torch.cuda.synchronize()
            assert out[0].item() == s_new and out[2].item() == n_new
            np.testing.assert_array_equal(out[1].cpu().numpy(), g_new)
            s, g, n = ctx.score_mi(coeff)
            assert s == s_new and n == n_new
            np.testing.assert_array_equal(g, g_new)
            del graph


def test_images_of_an_mse_context_cost_what_they_did():
    """b200bsp_set_images does nothing for the line kernel that a context
    pinned to the tile kernel does without (12 % of its time, when it formed
    pass 1's image of the moving bins)."""
    import time

    import torch
    fixed = synth.gaussian_blobs((256, 256, 96), seed=3)
    grid = BsplineGrid.for_volume(fixed, 8)
    img = torch.from_numpy(fixed.img).cuda()
    best = {}
    for _ in range(2):
        for kernel in ("tile", "auto"):
            with P.Context(fixed, fixed, grid, tc_kernel=kernel) as ctx:
                for _ in range(40):
                    torch.cuda.synchronize()
                    t0 = time.perf_counter()
                    ctx.set_images(img, img)
                    torch.cuda.synchronize()
                    best[kernel] = min(best.get(kernel, np.inf),
                                       time.perf_counter() - t0)
    assert best["auto"] < 1.06 * best["tile"], best


def _exact_gradient(fixed, moving, grid):
    """MSE gradient without a displacement, voxel on voxel, in 64 bits."""
    f, m = (v.img.astype(np.float64) for v in (fixed, moving))
    mg = P.volume_grad(moving).reshape(m.shape + (3,)).astype(np.float64)
    dc = (m - f)[..., None] * mg * (2.0 / f.size)
    for axis, v in ((2, grid.vox_per_rgn[0]), (1, grid.vox_per_rgn[1]),
                    (0, grid.vox_per_rgn[2])):
        n = dc.shape[axis]
        lut = O.port_basis_lut(v).reshape(v, 4).astype(np.float64)
        b = np.zeros((n, (n + v - 1) // v + 3))
        for i in range(n):
            b[i, i // v:i // v + 4] = lut[i % v]
        dc = np.moveaxis(np.tensordot(b, dc, axes=(0, axis)), 0, axis)
    return dc.reshape(-1)


@pytest.mark.parametrize("dim,vpr", [((64, 64, 64), (8, 8, 8)),
                                     ((100, 90, 80), (10, 10, 10)),
                                     ((72, 66, 60), (3, 3, 3)),
                                     ((150, 128, 70), (5, 6, 4))])
def test_gradient_sums_are_as_good_as_the_tile_kernels(dim, vpr):
    """Without a displacement every position is exact, so what is left of the
    gradient's error is its products and sums.  The line kernel sums some
    tens of products in float along each axis, where the tile kernel sums a
    tile's hundreds in float and the tiles in double: no further from 64 bits
    than that."""
    fixed = synth.gaussian_blobs(dim, spacing=(1, 1, 1), seed=12)
    moving = synth.gaussian_blobs(dim, spacing=(1, 1, 1), seed=13)
    grid = BsplineGrid.for_volume(fixed, vpr)
    want = _exact_gradient(fixed, moving, grid)
    err = {}
    for kernel in ("tile", "auto"):
        with P.Context(fixed, moving, grid, tc_kernel=kernel) as ctx:
            ctx.set_images()
            _, g, n = ctx.score_mse_f64(np.zeros(grid.num_coeff, np.float32))
        assert n == fixed.img.size
        err[kernel] = rel_err(g, want)
    print(err)
    assert err["auto"] <= err["tile"] < 1e-5, err
