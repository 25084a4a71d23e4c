"""The tensor-core kernels that the optimiser's evaluations run, and that
evaluations of their own reach only where the line kernel does not: pinned
(b200bsp_opts.tc_kernel) against the double-precision oracle, and as the
optimiser itself runs them.

Bars as for the evaluations of the default contexts: score relative 1e-5,
gradient relative L2 1e-3, histograms relative L2 1e-5, voxel count within
0.01 % (+2).
"""
import numpy as np
import pytest

import oracle as O
import plastimatch_b200 as P
from conftest import (ROI_TAGS, golden_names, load_golden, load_rois,
                      pick_rois, rel_err)
from plastimatch_b200 import synth
from plastimatch_b200.geometry import BsplineGrid, Volume

pytestmark = pytest.mark.gpu

ROTATED = (0.0, 1.0, 0.0, -1.0, 0.0, 0.0, 0.0, 0.0, 1.0)


def _check(s, g, n, f64):
    assert abs(n - f64.num_vox) <= 1e-4 * f64.num_vox + 2, (n, f64.num_vox)
    assert abs(s - f64.score) <= 1e-5 * abs(f64.score), (s, f64.score)
    assert rel_err(g, f64.grad) < 1e-3, rel_err(g, f64.grad)


def _case(shape=(48, 40, 36), vpr=(6, 5, 4), seed=61, dcos=None, roi=None,
          remap=True):
    fixed = synth.gaussian_blobs(shape, spacing=(1.0, 1.2, 1.5), seed=seed)
    g0 = BsplineGrid.for_volume(fixed, 8)
    moving = synth.warp_trilinear(fixed, fixed, g0,
                                  synth.random_coeff(g0, 1.5, seed + 1))
    if remap:
        moving = synth.intensity_remap(moving, 0.7, 5.0, seed + 2)
    if dcos is not None:
        fixed, moving = (Volume(v.img, origin=v.origin, spacing=v.spacing,
                                dcos=dcos) for v in (fixed, moving))
    kw = {} if roi is None else dict(roi_offset=roi[0], roi_dim=roi[1])
    grid = BsplineGrid.for_volume(fixed, vpr, **kw)
    return fixed, moving, grid, synth.random_coeff(grid, 1.0, seed + 3)


@pytest.mark.parametrize("name", golden_names("mi"))
def test_tile_kernel_pvi8_golden(name):
    fixed, moving, grid, coeff, rec = load_golden(name)
    with P.Context(fixed, moving, grid, tc_kernel="tile", mi_bins=32) as ctx:
        ctx.set_images()
        s, g, n, (fh, mh, jh) = ctx.score_mi(coeff, with_hist=True)
    f64 = O.port_mi(grid, fixed, moving, coeff, bins=32, precision="f64")
    _check(s, g, n, f64)
    assert rel_err(g, rec["mi_grad"]) < 1e-3
    assert rel_err(fh, rec["f_hist"]) < 1e-5
    assert rel_err(mh, rec["m_hist"]) < 1e-5
    assert rel_err(jh, rec["j_hist"]) < 1e-5


@pytest.mark.parametrize("kernel", ["tile", "xlane"])
@pytest.mark.parametrize("bins", [16, 32])
@pytest.mark.parametrize("case", [
    dict(), dict(vpr=(8, 8, 8)), dict(dcos=ROTATED),
    dict(roi=((4, 3, 2), (36, 30, 28)))])
def test_pinned_parzen(case, bins, kernel):
    fixed, moving, grid, coeff = _case(**case)
    with P.Context(fixed, moving, grid, tc_kernel=kernel, mi_bins=bins,
                   mi_window="parzen") as ctx:
        ctx.set_images()
        s, g, n, (fh, mh, jh) = ctx.score_mi(coeff, with_hist=True)
    ref = O.port_mi_parzen(grid, fixed, moving, coeff, bins=bins)
    _check(s, g, n, ref)
    assert rel_err(jh, ref.j_hist) < 1e-5
    assert rel_err(mh, ref.m_hist) < 1e-5
    assert rel_err(fh, ref.f_hist) < 1e-5


@pytest.mark.parametrize("kernel", ["tile", "xlane"])
@pytest.mark.parametrize("case", [
    dict(), dict(vpr=(8, 8, 8)), dict(vpr=(5, 5, 5), dcos=ROTATED)])
def test_pinned_trilinear_gradient(case, kernel):
    fixed, moving, grid, coeff = _case(remap=False, **case)
    with P.Context(fixed, moving, grid, tc_kernel=kernel,
                   mse_grad="trilinear") as ctx:
        ctx.set_images()
        out = ctx.score_mse(coeff)
    _check(*out, O.port_mse(grid, fixed, moving, coeff, grad_mode=1,
                            precision="f64"))


@pytest.mark.parametrize("grad", ["nearest", "trilinear"])
@pytest.mark.parametrize("tag", ROI_TAGS)
@pytest.mark.parametrize("name", golden_names("roimask_mse"))
def test_xlane_kernel_rois(name, tag, grad):
    fixed, moving, grid, coeff, rec = load_golden(name)
    fr, mr = pick_rois(tag, *load_rois(rec))
    with P.Context(fixed, moving, grid, tc_kernel="xlane",
                   mse_grad=grad) as ctx:
        if grad == "nearest":
            ctx.set_images(moving_grad=rec["moving_grad"])
        else:
            ctx.set_images()
        ctx.set_roi(fr, mr)
        assert ctx.mse_kernel()[0] == "xlane"
        out = ctx.score_mse(coeff)
    kw = (dict(moving_grad=rec["moving_grad"]) if grad == "nearest"
          else dict(grad_mode=1))
    _check(*out, O.port_mse(grid, fixed, moving, coeff, precision="f64",
                            fixed_roi=fr, moving_roi=mr, **kw))


@pytest.mark.parametrize("shape,vpr", [((96, 80, 48), (12, 5, 5)),
                                       ((200, 64, 40), (11, 4, 4))])
def test_autotuned_split_keeps_parity(shape, vpr):
    """On a grid that the line kernel refuses, the evaluations run on the
    kernel and split that the autotuner picked."""
    fixed, moving, grid, coeff = _case(shape, vpr, remap=False)
    with P.Context(fixed, moving, grid) as ctx:
        ctx.set_images()
        t = ctx.autotune(coeff, evals=2)
        name, tiles, _ = ctx.mse_kernel()
        assert name in ("tile", "xlane") and tiles == t
        s, g, n = ctx.score_mse(coeff)
        s2, g2, n2 = ctx.score_mse(coeff)
    _check(s, g, n, O.port_mse(grid, fixed, moving, coeff,
                               moving_grad=O.port_volume_grad(moving),
                               precision="f64"))
    assert s == s2 and n == n2
    np.testing.assert_array_equal(g, g2)


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("what", ["mse", "roi", "pvi8", "parzen"])
def test_optimiser_score_is_the_oracles(what, autotune):
    """The score that a short run returns, at the coefficients that it
    returns with it (the last evaluated ones), on a grid that the line kernel
    takes: every one of these kernels as the optimiser runs it."""
    if what == "roi":
        fixed, moving, grid, coeff, rec = load_golden("roimask_mse_small")
        fr, mr = load_rois(rec)
    else:
        fixed, moving, grid, coeff = _case(remap=what != "mse")
    metric = "mse" if what in ("mse", "roi") else "mi"
    kw = {} if metric == "mse" else dict(mi_window=what)
    with P.Context(fixed, moving, grid, **kw) as ctx:
        assert ctx.mse_kernel()[0] == "line"
        ctx.set_images()
        if what == "roi":
            ctx.set_roi(fr, mr)
        if autotune:
            ctx.autotune(coeff, evals=1)
        c, res = ctx.optimize_lbfgs(coeff, metric=metric, max_its=3,
                                    max_feval=8)
    assert res["fevals"] >= 3 and not np.array_equal(c, coeff)
    if what == "pvi8":
        f64 = O.port_mi(grid, fixed, moving, c, bins=32, precision="f64")
    elif what == "parzen":
        f64 = O.port_mi_parzen(grid, fixed, moving, c, bins=32)
    else:
        rois = dict(fixed_roi=fr, moving_roi=mr) if what == "roi" else {}
        f64 = O.port_mse(grid, fixed, moving, c, precision="f64",
                         moving_grad=O.port_volume_grad(moving), **rois)
    assert abs(res["score"] - f64.score) <= 1e-5 * abs(f64.score)
