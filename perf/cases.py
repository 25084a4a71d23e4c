"""The work that a registration program has this library do, as cases that can
be timed and compared: cost-function evaluations (MSE and Mattes MI, with
their gradients) over the sizes, grids and options that registrations use,
several registrations evaluated together, a short registration, and the
warp that ends one.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  contexts, images and coefficients on the GPU
    run(state)           one pass through the public entry points
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    what run returns, in 64 bits, from plain torch
"""
import math

import numpy as np
import torch

import plastimatch_b200 as P
from plastimatch_b200.geometry import BsplineGrid, Roi, Volume

DEV = "cuda"


# ---- the cases ----------------------------------------------------------------
#
# A case: "kind" (what is called), the fixed image's dims nx, ny, nz and
# spacing sx, sy, sz (mm), the moving image's dims as the fixed one's plus
# px, py, pz voxels (half of them before its first voxel), voxels per
# control-grid region vx, vy, vz, rotation of both images about z ("angle",
# degrees), and what else the kind takes.

def _case(kind, dim, spacing, vpr, name=None, pad=(0, 0, 0), angle=0.0, **kw):
    c = {"kind": kind, "nx": dim[0], "ny": dim[1], "nz": dim[2],
         "sx": spacing[0], "sy": spacing[1], "sz": spacing[2],
         "px": pad[0], "py": pad[1], "pz": pad[2],
         "vx": vpr[0], "vy": vpr[1], "vz": vpr[2], "angle": angle}
    c.update(kw)
    if name:
        c["name"] = name
    return c


MARGIN = (24, 24, 16)      # a moving scan that covers more than the fixed one


def listed():
    return [
        # The smallest registration (the reference's CPU-runnable case), on
        # the device: launches and latency are what it costs.
        _case("mse", (64, 64, 64), (1.0, 1.0, 1.0), (8, 8, 8),
              "mse_64_vpr8", grad="nearest"),
        # A cropped scan in patient axes: odd sizes, the last tiles ragged on
        # every axis, rotated direction cosines, a moving image of other
        # dims.
        _case("mse", (131, 117, 83), (1.17, 1.17, 1.5), (6, 6, 6),
              "mse_131x117x83_vpr6_oblique", pad=(-6, 5, 4), angle=12.0,
              grad="nearest"),
        # The cost function of one iteration at the benchmark's size.
        _case("mse", (256, 256, 128), (0.98, 0.98, 2.5), (5, 5, 5),
              "mse_256x256x128_vpr5", grad="nearest"),
        # The finest level of a full-resolution scan.
        _case("mse", (512, 512, 160), (1.0, 1.0, 2.5), (10, 10, 4),
              "mse_512x512x160_vpr10x10x4", grad="nearest"),
        # The whole cost function with the curvature regulariser, host
        # arrays in and out, as an optimiser on the host calls it, with the
        # derivative of the trilinear interpolant (the one that agrees with
        # finite differences).
        _case("score", (128, 128, 96), (1.0, 1.0, 1.0), (6, 6, 6),
              "score_128x128x96_vpr6_curvature", grad="trilinear",
              curvature=0.005),
        # A registration inside a body mask.
        _case("mse_roi", (200, 180, 90), (1.0, 1.0, 2.0), (7, 7, 4),
              "mse_roi_200x180x90_vpr7x7x4", grad="nearest"),
        # Multi-modal registration with the reference's histograms, at the
        # benchmark's size.
        _case("mi", (256, 256, 128), (0.98, 0.98, 2.5), (5, 5, 5),
              "mi_pvi8_256x256x128_vpr5", pad=MARGIN, window="pvi8", bins=32),
        # The coarsest and the middle level of the multi-modal pyramid over
        # a 512x512x160 scan (Parzen windows).
        _case("mi", (128, 128, 40), (2.5, 2.5, 2.5), (4, 4, 4),
              "mi_parzen_128x128x40_vpr4", pad=MARGIN, window="parzen",
              bins=32),
        _case("mi", (256, 256, 80), (2.0, 2.0, 2.5), (5, 5, 4),
              "mi_parzen_256x256x80_vpr5x5x4", pad=MARGIN, window="parzen",
              bins=32),
        # Multi-atlas: registrations of uneven sizes evaluated together.
        _case("batch", (160, 144, 80), (1.5, 1.5, 2.0), (7, 7, 5),
              "batch_8", grad="nearest", count=8),
        # A short registration: the optimiser with everything that it calls.
        _case("lbfgs", (64, 64, 64), (1.0, 1.0, 1.0), (8, 8, 8),
              "lbfgs_64_vpr8_4_iterations", grad="trilinear", its=4),
        # The moving image carried onto the fixed grid at a registration's
        # end.
        _case("warp", (256, 256, 128), (0.98, 0.98, 2.5), (5, 5, 5),
              "warp_256x256x128_vpr5", pad=MARGIN),
    ]


def draw(rng):
    """One more case: 2^18 to 2^25 voxels, in-plane dims of the same order,
    1 to 2.5 mm voxels, regions of 4 to 10 voxels (at most 1000 in all)."""
    kind = rng.choice(["mse", "mse", "mse", "mi", "mi", "score", "mse_roi",
                       "batch", "lbfgs", "warp"])
    top = {"lbfgs": 19.0, "batch": 20.5, "score": 22.5, "mi": 23.5}.get(kind, 25.0)
    n = 2.0 ** rng.uniform(18.0, top)
    aspect = rng.uniform(1.0, 3.2)                       # in-plane / through-plane
    nz = (n / aspect ** 2) ** (1.0 / 3.0)
    nxy = math.sqrt(n / nz)
    skew = rng.uniform(0.85, 1.18)
    dim = tuple(max(24, int(v)) for v in (nxy * skew, nxy / skew, nz))
    vpr = tuple(rng.randint(4, 10) for _ in range(3))
    if kind in ("mse_roi", "score"):
        sp = rng.choice([1.0, 2.0])
        sp = (sp, sp, sp if kind == "score" else rng.choice([1.0, 2.0]))
        vpr = (vpr[0],) * 3 if kind == "score" else vpr
    else:
        s = round(rng.uniform(1.0, 2.5), 2)
        sp = (s, s, round(rng.uniform(1.0, 2.5), 2))
    angle = round(rng.uniform(-20.0, 20.0), 1) if kind == "mse" and rng.random() < 0.3 else 0.0
    kw = {}
    pad = (0, 0, 0)
    if kind == "mi":
        kw = {"window": rng.choice(["pvi8", "parzen"]), "bins": rng.choice([20, 32, 48])}
        pad = MARGIN
    elif kind == "warp":
        pad = MARGIN
    else:
        kw["grad"] = rng.choice(["nearest", "nearest", "trilinear"])
        if kind == "mse":
            pad = tuple(rng.randint(-6, 10) for _ in range(3))
    if kind == "score":
        kw["curvature"] = 0.005
    elif kind == "batch":
        kw["count"] = rng.randint(3, 8)
    elif kind == "lbfgs":
        kw.update(grad="trilinear", its=rng.randint(2, 4))
    return _case(kind, dim, sp, vpr, pad=pad, angle=angle, **kw)


# ---- inputs -------------------------------------------------------------------

def _parts(case):
    """The registrations of a case: one, or a batch's uneven ones."""
    if case["kind"] != "batch":
        return [case]
    out = []
    for k in range(case["count"]):
        f = (1.0 + 0.5 * math.sin(1.0 + 2.3 * k), 1.0 + 0.4 * math.sin(0.4 + 1.7 * k),
             1.0 + 0.4 * math.cos(0.3 + 1.1 * k))
        c = dict(case, kind="mse")
        for d, q in zip("xyz", f):
            c["n" + d] = max(24, int(case["n" + d] * q))
        out.append(c)
    return out


def _geometry(case):
    """(fixed, moving, grid) with empty images."""
    dim = [case["n" + d] for d in "xyz"]
    pad = [case["p" + d] for d in "xyz"]
    sp = tuple(case["s" + d] for d in "xyz")
    a = math.radians(case["angle"])
    dcos = (math.cos(a), -math.sin(a), 0.0, math.sin(a), math.cos(a), 0.0, 0.0, 0.0, 1.0)
    mdim = [n + p for n, p in zip(dim, pad)]
    # an ROI case's origin keeps voxel positions exact, so that the voxels of
    # its masks are the same in any arithmetic
    shift = (0.0, 0.0, 0.0) if case["kind"] == "mse_roi" else (0.37, -0.21, 0.55)
    off = np.array([s - (p // 2) * q for s, p, q in zip(shift, pad, sp)])
    origin = tuple(float(v) for v in np.array(dcos).reshape(3, 3) @ off)

    def vol(d, o):
        return Volume(np.zeros((d[2], d[1], d[0]), np.float32), origin=o, spacing=sp, dcos=dcos)
    fixed = vol(dim, (0.0, 0.0, 0.0))
    grid = BsplineGrid.for_volume(fixed, tuple(case["v" + d] for d in "xyz"))
    return fixed, vol(mdim, origin), grid


def _smooth(img):
    """What a scanner's point spread leaves: [1 4 6 4 1] / 16 per axis."""
    for d in range(3):
        for _ in range(2):
            n = img.shape[d]
            lo = torch.cat([img.narrow(d, 0, 1), img.narrow(d, 0, n - 1)], d)
            hi = torch.cat([img.narrow(d, 1, n - 1), img.narrow(d, n - 1, 1)], d)
            img = 0.25 * lo + 0.5 * img + 0.25 * hi
    return img


def _image(dim, centres, sigmas, amps, gen):
    """Soft-tissue-like content in air, as a registration smooths it before it
    starts: structures of a few to some tens of voxels, and correlated noise
    of a few grey levels."""
    e = [torch.exp(-0.5 * ((torch.arange(dim[d], device=DEV)[None, :] - centres[:, d:d + 1])
                           / sigmas[:, d:d + 1]) ** 2) for d in range(3)]
    zy = (e[2] * amps[:, None])[:, :, None] * e[1][:, None, :]
    img = torch.einsum("bzy,bx->zyx", zy, e[0])
    w = torch.randn(dim[2], dim[1], dim[0], generator=gen, device=DEV)
    for _ in range(4):
        w = _smooth(w)
    return img.add_(w, alpha=float(3.0 / w.std())).contiguous()


def _inputs(case, seed):
    """(fixed image, moving image, coefficients) on the GPU."""
    fixed, moving, grid = _geometry(case)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    n = 40
    dim = torch.tensor(fixed.dim, device=DEV, dtype=torch.float32)
    u = torch.rand(n, 5, generator=gen, device=DEV)
    centres = (0.25 + 0.5 * u[:, :3]) * dim
    sigmas = (0.07 + 0.07 * u[:, 3:4]) * dim
    amps = 100.0 + 900.0 * u[:, 4]
    # the moving anatomy: displaced by a voxel or so, grown or shrunk a little
    j = torch.randn(n, 4, generator=gen, device=DEV)
    half = torch.tensor([case["p" + d] // 2 for d in "xyz"], device=DEV, dtype=torch.float32)
    f = _image(fixed.dim, centres, sigmas, amps, gen)
    m = _image(moving.dim, centres + 1.2 * j[:, :3] + half, sigmas * (1.0 + 0.03 * j[:, 3:4]),
               amps, gen)
    if case["kind"] == "mi":       # another modality: a nonlinear remap
        lo, hi = m.min(), m.max()
        m = (lo + (hi - lo) * ((m - lo) / (hi - lo)) ** 0.7).contiguous()
    # mid-run coefficients of half a millimetre; a registration starts at none
    c = torch.randn(grid.num_coeff, generator=gen, device=DEV)
    return f, m, c * (0.0 if case["kind"] == "lbfgs" else 0.5)


def _masks(case, fixed, moving):
    """An ellipsoid body mask on each image (uint8, z y x)."""
    def ell(v, q):
        nx, ny, nz = v.dim
        g = [((np.arange(n) - 0.5 * n) / (q * n)) ** 2 for n in (nx, ny, nz)]
        return ((g[2][:, None, None] + g[1][None, :, None] + g[0][None, None, :]) <= 1.0).astype(np.uint8)
    return ell(fixed, 0.40), ell(moving, 0.47)


# ---- one pass -----------------------------------------------------------------

_stream = None


def _program_stream():
    """The stream that the program orders its work on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case, "ctx": [], "coeff": [], "grad": []}
    for k, c in enumerate(_parts(case)):
        fixed, moving, grid = _geometry(c)
        f, m, coeff = _inputs(c, seed + 1000 * k)
        opts = {"mse_grad": c.get("grad", "nearest")}
        if kind == "mi":
            opts.update(mi_window=c["window"], mi_bins=c["bins"])
        ctx = P.Context(fixed, moving, grid, **opts)
        ctx.set_stream(_program_stream())
        torch.cuda.synchronize()
        ctx.set_images(f, m)
        if kind == "mse_roi":
            fm, mm = _masks(c, fixed, moving)
            ctx.set_roi(Roi.like(fixed, fm), Roi.like(moving, mm))
        state["ctx"].append(ctx)
        state["coeff"].append(coeff)
        state["grad"].append(torch.zeros(grid.num_coeff, device=DEV))
    state["score"] = torch.zeros(len(state["ctx"]), device=DEV)
    if kind in ("score", "mi", "lbfgs"):
        state["host"] = state["coeff"][0].cpu().numpy()
    if kind == "score":
        state["reg"] = P.reg_parms(curvature=case["curvature"])
    if kind == "batch":
        state["batch"] = P.Batch(state["ctx"])
    if kind == "warp":
        nx, ny, nz = fixed.dim
        state["out"] = torch.zeros(nz, ny, nx, device=DEV)
    return state


def run(state):
    kind, ctx = state["kind"], state["ctx"][0]
    if kind in ("mse", "mse_roi"):
        s, g, _ = ctx.score_mse(state["coeff"][0], state["grad"][0], state["score"])
        return {"score": s, "grad": g}
    if kind == "score":
        total, grad, smetric, _ = ctx.score(state["host"], lam=1.0, reg=state["reg"])
        return {"total": total, "grad": grad, "smetric": smetric}
    if kind == "mi":
        s, g, n = ctx.score_mi(state["host"])
        return {"score": s, "grad": g, "num_vox": n}
    if kind == "batch":
        state["batch"].score_mse(state["coeff"], state["grad"], state["score"])
        return {"score": state["score"], "grad": state["grad"]}
    if kind == "lbfgs":
        c, res = ctx.optimize_lbfgs(state["host"], max_its=state["case"]["its"], max_feval=40)
        return {"coeff": c, "score": res["score"], "fevals": res["fevals"]}
    rc = P.lib().b200bsp_warp(ctx._h, state["coeff"][0].data_ptr(), -1000.0,
                              state["out"].data_ptr())
    if rc:
        raise P.B200Error(rc, "warp")
    return state["out"]


def work(case):
    """Both images once and the coefficients and outputs once (the moving
    gradient follows from the moving image); per voxel the separable field
    and adjoint along one axis, the trilinear sample and its derivative."""
    by = fl = 0.0
    for c in _parts(case):
        fixed, moving, grid = _geometry(c)
        n = float(fixed.npix)
        knots = 4.0 * grid.num_coeff
        if c["kind"] == "warp":
            by += 4.0 * n + 4.0 * moving.npix + knots
            fl += n * 50.0
            continue
        by += 4.0 * n + 4.0 * moving.npix + 2.0 * knots
        fl += n * (130.0 if c["kind"] == "mi" else 90.0)
    if case["kind"] == "lbfgs":
        by, fl = by * (case["its"] + 2), fl * (case["its"] + 2)
    return {"bytes": by, "flops": fl}


# ---- the same in 64 bits --------------------------------------------------------

def _basis(n, v, d=torch.float64):
    """[n voxels, knots] weights of the cubic B-spline with v voxels a region."""
    i = torch.arange(n, device=DEV)
    p, u = i // v, (i % v).to(d) / v
    w = torch.stack([(1 - u) ** 3 / 6, (3 * u ** 3 - 6 * u ** 2 + 4) / 6,
                     (-3 * u ** 3 + 3 * u ** 2 + 3 * u + 1) / 6, u ** 3 / 6], 1)
    out = torch.zeros(n, (n - 1) // v + 4, dtype=d, device=DEV)
    for k in range(4):
        out[i, p + k] = w[:, k]
    return out


class _Exact:
    """One registration's evaluation in float64, slab by slab along z."""

    def __init__(self, case, seed):
        self.case = case
        self.fixed, self.moving, self.grid = _geometry(case)
        f, m, c = _inputs(case, seed)
        self.f, self.m, self.c = f.double(), m.double(), c.double()
        dim, vpr = self.fixed.dim, self.grid.vox_per_rgn
        self.B = [_basis(dim[d], vpr[d]) for d in range(3)]
        as64 = lambda v: torch.tensor(np.asarray(v, np.float64), device=DEV)  # noqa: E731
        fdc = as64(self.fixed.dcos).reshape(3, 3)
        sp = as64(self.fixed.spacing)
        self.step = fdc * sp[None, :]
        self.inv = torch.linalg.inv(as64(self.moving.dcos).reshape(3, 3))
        self.msp = as64(self.moving.spacing)
        self.proj = self.inv / self.msp[:, None]
        self.fo, self.mo = as64(self.fixed.origin), as64(self.moving.origin)
        self.masks = None
        if case["kind"] == "mse_roi":
            self.masks = [torch.from_numpy(q).to(DEV).reshape(-1) for q in
                          _masks(case, self.fixed, self.moving)]

    def slabs(self):
        nx, ny, nz = self.fixed.dim
        h = max(1, int(3e6) // (nx * ny))
        return [(z, min(nz, z + h)) for z in range(0, nz, h)]

    def locate(self, z0, z1):
        """Field, inside test, corner and fractions of the slab's voxels."""
        nx, ny, _ = self.fixed.dim
        cx, cy, cz = self.grid.cdims
        C = self.c.reshape(cz, cy, cx, 3)
        e = torch.einsum("zk,kjic->zjic", self.B[2][z0:z1], C)
        e = torch.einsum("yj,zjic->zyic", self.B[1], e)
        d = torch.einsum("xi,zyic->zyxc", self.B[0], e)
        ijk = torch.stack(torch.meshgrid(
            torch.arange(z0, z1, device=DEV), torch.arange(ny, device=DEV),
            torch.arange(nx, device=DEV), indexing="ij")[::-1], -1).double()
        pos = self.fo + ijk @ self.step.T + d
        ma = ((pos - self.mo) @ self.proj.T).reshape(-1, 3)
        hi = torch.tensor(self.moving.dim, device=DEV)
        ok = ((ma > -0.5) & (ma < hi - 0.5)).all(1)
        if self.masks is not None:
            q = torch.minimum(ma.floor().clamp(min=0).long(), hi - 1)
            ok &= self.masks[1][q[:, 0] + hi[0] * (q[:, 1] + hi[1] * q[:, 2])] != 0
            ok &= self.masks[0][z0 * nx * ny:z1 * nx * ny] != 0
        fl = torch.minimum(ma.floor().clamp(min=0), (hi - 2).double())
        w = (ma - fl).clamp(0, 1)
        clamped = (ma < 0) | (ma >= hi - 1)
        return ok, fl.long(), w, clamped

    def corners(self, img, fl):
        nx, ny, _ = self.moving.dim
        i = fl[:, 0] + nx * (fl[:, 1] + ny * fl[:, 2])
        flat = img.reshape(-1)
        return [flat[i + (k & 1) + nx * (k >> 1 & 1) + nx * ny * (k >> 2)] for k in range(8)]

    @staticmethod
    def weights(w):
        a = torch.stack([1 - w, w])
        return [a[k & 1][:, 0] * a[k >> 1 & 1][:, 1] * a[k >> 2][:, 2] for k in range(8)]

    @staticmethod
    def index_grad(w, m):
        """Index-space derivative of the trilinear interpolant of corners m."""
        a = torch.stack([1 - w, w])
        s = (-1.0, 1.0)
        gx = sum(s[k & 1] * a[k >> 1 & 1][:, 1] * a[k >> 2][:, 2] * m[k] for k in range(8))
        gy = sum(a[k & 1][:, 0] * s[k >> 1 & 1] * a[k >> 2][:, 2] * m[k] for k in range(8))
        gz = sum(a[k & 1][:, 0] * a[k >> 1 & 1][:, 1] * s[k >> 2] * m[k] for k in range(8))
        return torch.stack([gx, gy, gz], 1)

    def adjoint(self, dc, z0, z1):
        nx, ny, _ = self.fixed.dim
        g = torch.einsum("xi,zyxc->zyic", self.B[0], dc.reshape(z1 - z0, ny, nx, 3))
        g = torch.einsum("yj,zyic->zjic", self.B[1], g)
        return torch.einsum("zk,zjic->kjic", self.B[2][z0:z1], g)

    def gradient_image(self):
        """Central differences with replicated borders, turned into world axes."""
        out = []
        for d in range(3):
            ax, n = 2 - d, self.moving.dim[d]
            lo = torch.cat([self.m.narrow(ax, 0, 1), self.m.narrow(ax, 0, n - 1)], ax)
            hi = torch.cat([self.m.narrow(ax, 1, n - 1), self.m.narrow(ax, n - 1, 1)], ax)
            out.append((hi - lo) / 2.0 / self.msp[d])
        return torch.stack(out, -1).reshape(-1, 3) @ self.inv.T

    def mse(self):
        nx, ny, nz = self.fixed.dim
        mx, my, _ = self.moving.dim
        nearest = self.case["grad"] == "nearest"
        gimg = self.gradient_image() if nearest else None
        score, count, grad = 0.0, 0, 0.0
        for z0, z1 in self.slabs():
            ok, fl, w, _ = self.locate(z0, z1)
            m = self.corners(self.m, fl)
            v = sum(a * b for a, b in zip(self.weights(w), m))
            diff = torch.where(ok, v - self.f[z0:z1].reshape(-1), 0.0)
            if nearest:
                r = fl + (w >= 0.5)
                g = gimg[r[:, 0] + mx * (r[:, 1] + my * r[:, 2])]
            else:
                g = self.index_grad(w, m) / self.msp
            score = score + (diff * diff).sum()
            count += int(ok.sum())
            grad = grad + self.adjoint(diff[:, None] * g, z0, z1)
        return score / count, (2.0 / count * grad).reshape(-1)

    def mi_pvi8(self):
        bins = self.case["bins"]

        def binned(img):
            lo, hi = img.min(), img.max()
            delta = (hi - lo) / (bins - 1)
            return ((img - (lo - 0.5 * delta)) / delta).floor().long().clamp(0, bins - 1)
        fb, mb = binned(self.f), binned(self.m)
        joint = torch.zeros(bins * bins, dtype=torch.float64, device=DEV)
        n = 0
        for z0, z1 in self.slabs():
            ok, fl, w, _ = self.locate(z0, z1)
            f = fb[z0:z1].reshape(-1)
            for b, q in zip(self.corners(mb, fl), self.weights(w)):
                joint.index_add_(0, f * bins + b, torch.where(ok, q, 0.0))
            n += int(ok.sum())
        j = joint.reshape(bins, bins)
        pf, pm = j.sum(1, keepdim=True), j.sum(0, keepdim=True)
        ratio = torch.log((n * j / (pf * pm)).clamp(min=1e-300))
        score = -(torch.where(j > 0.001 / bins ** 2, j * ratio, 0.0)).sum() / n
        table = torch.where(j > 0.0001, ratio - score, 0.0).reshape(-1)
        grad = 0.0
        for z0, z1 in self.slabs():
            ok, fl, w, _ = self.locate(z0, z1)
            f = fb[z0:z1].reshape(-1)
            t = [table[f * bins + b] for b in self.corners(mb, fl)]
            d = -self.index_grad(w, t) / n
            # world axes row by row, each row on what the rows above left
            # (the reference's order)
            p = self.proj
            d0 = d @ p[0]
            d1 = d0 * p[1, 0] + d[:, 1] * p[1, 1] + d[:, 2] * p[1, 2]
            d2 = d0 * p[2, 0] + d1 * p[2, 1] + d[:, 2] * p[2, 2]
            d = torch.where(ok[:, None], torch.stack([d0, d1, d2], 1), 0.0)
            grad = grad + self.adjoint(d, z0, z1)
        return score, grad.reshape(-1), n

    def mi_parzen(self):
        bins = self.case["bins"]
        lo, hi = self.f.min(), self.f.max()
        fb = (((self.f - lo) / ((hi - lo) / (bins - 4))).floor().long() + 2).clamp(2, bins - 3)
        mlo, mdelta = self.m.min(), (self.m.max() - self.m.min()) / (bins - 4)

        def window(z0, z1):
            ok, fl, w, clamped = self.locate(z0, z1)
            m = self.corners(self.m, fl)
            u = (sum(a * b for a, b in zip(self.weights(w), m)) - mlo) / mdelta + 2.0
            k0 = u.floor().long().clamp(1, bins - 3) - 1
            return ok, w, clamped, m, u, k0, fb[z0:z1].reshape(-1)

        def b3(t):
            a = t.abs()
            return torch.where(a < 1, 2 / 3 - a * a + 0.5 * a ** 3,
                               torch.where(a < 2, (2 - a) ** 3 / 6, 0.0))

        def b3d(t):
            a = t.abs()
            return torch.where(a < 1, -2 * t + 1.5 * t * a,
                               torch.where(a < 2, -0.5 * t.sign() * (2 - a) ** 2, 0.0))
        joint = torch.zeros(bins * bins, dtype=torch.float64, device=DEV)
        n = 0
        for z0, z1 in self.slabs():
            ok, _, _, _, u, k0, f = window(z0, z1)
            for k in range(4):
                joint.index_add_(0, f * bins + k0 + k, torch.where(ok, b3(k0 + k - u), 0.0))
            n += int(ok.sum())
        p = joint.reshape(bins, bins) / n
        pf, pm = p.sum(1, keepdim=True), p.sum(0, keepdim=True)
        # weights are held in 2^-24 units: smaller sums are none at all
        live = joint.reshape(bins, bins) > 2.0 ** -25
        safe = torch.where(live, p, 1.0)
        score = -torch.where(live, p * torch.log(safe / (pf * pm).clamp(min=1e-300)), 0.0).sum()
        table = torch.where(live, torch.log(safe / pm.clamp(min=1e-300)), 0.0).reshape(-1)
        grad = 0.0
        for z0, z1 in self.slabs():
            ok, w, clamped, m, u, k0, f = window(z0, z1)
            s = sum(b3d(k0 + k - u) * table[f * bins + k0 + k] for k in range(4)) / (n * mdelta)
            g = torch.where(clamped, 0.0, self.index_grad(w, m)) @ self.proj
            grad = grad + self.adjoint(torch.where(ok[:, None], s[:, None] * g, 0.0), z0, z1)
        return score, grad.reshape(-1), n

    def curvature(self, penalty):
        """Integral of the squared second derivatives (each mixed one once),
        and its gradient; regions of equal edges."""
        cx, cy, cz = self.grid.cdims
        h = float(self.grid.vox_per_rgn[0] * self.fixed.spacing[0])
        poly = torch.tensor([[1, -3, 3, -1], [4, 0, -6, 3], [1, 3, 3, -3], [0, 0, 0, 1]],
                            dtype=torch.float64) / 6.0

        def gram(n, order):
            q = poly.clone()
            for _ in range(order):
                q = torch.cat([q[:, 1:] * torch.arange(1, 4, dtype=torch.float64),
                               torch.zeros(4, 1, dtype=torch.float64)], 1) / h
            pw = torch.arange(4)
            H = h / (pw[:, None] + pw[None, :] + 1.0).double()
            e = q @ H @ q.T
            G = torch.zeros(n, n, dtype=torch.float64)
            for t in range(n - 3):
                G[t:t + 4, t:t + 4] += e
            return G.to(DEV)
        G = [[gram(n, o) for o in range(3)] for n in (cx, cy, cz)]
        C = self.c.reshape(cz, cy, cx, 3)
        K = 0.0
        for o in ((2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)):
            t = torch.einsum("ab,zybc->zyac", G[0][o[0]], C)
            t = torch.einsum("ab,zbxc->zaxc", G[1][o[1]], t)
            K = K + torch.einsum("ab,byxc->ayxc", G[2][o[2]], t)
        K = penalty * K.reshape(-1)
        return (K * self.c).sum(), 2.0 * K

    def warp(self):
        out = []
        for z0, z1 in self.slabs():
            ok, fl, w, _ = self.locate(z0, z1)
            v = sum(a * b for a, b in zip(self.weights(w), self.corners(self.m, fl)))
            out.append(torch.where(ok, v, -1000.0))
        return torch.cat(out).reshape(self.f.shape)


def exact(case, seed):
    kind = case["kind"]
    if kind == "lbfgs":
        return None                      # a run of many evaluations: no closed value
    if kind == "batch":
        got = [_Exact(c, seed + 1000 * k).mse() for k, c in enumerate(_parts(case))]
        return {"score": torch.stack([s for s, _ in got]), "grad": [g for _, g in got]}
    x = _Exact(case, seed)
    if kind == "warp":
        return x.warp()
    if kind == "mi":
        s, g, n = x.mi_pvi8() if case["window"] == "pvi8" else x.mi_parzen()
        return {"score": s, "grad": g, "num_vox": n}
    s, g = x.mse()
    if kind == "score":
        r, rg = x.curvature(case["curvature"])
        return {"total": s + r, "grad": g + rg, "smetric": s}
    return {"score": s.reshape(1), "grad": g}
