"""The calls that a localisation program makes of bsfit, as cases to be timed.

A case names a workload and its sizes; ``prepare`` makes what such a program
holds before the call (ROIs or frames, the PSF model), ``run`` is the call
through the package's public entry points, ``work`` counts the bytes and
operations it cannot do without, and ``exact`` gives its outputs from plain
torch in 64 bits, where they have a value that does not hang on rounding.

Workloads ("kind"):
  fit     one device-resident fit call: fit type 6 (3D), 7 (4D colour), 8 (5D
          orientation) or 9 (4Pi), in single precision, double-float
          ("parity") or double ("f64"), sCMOS or several starts where asked
  host    the drop-in call on host arrays, GPUmleFit_LM_multiD (fit type 6)
  batch   one batched fit of three ROI sizes (fit type 6)
  frames  camera frames to ROIs (find_rois_torch)
  coeffs  B-spline coefficients of a sampled PSF stack (bsarray_coeffs_torch)
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gpu-based-b-spline-fitter_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bsfit  # noqa: E402
from bsfit import workloads as wl  # noqa: E402

ITERATIONS = {6: 30, 7: 60, 8: 60, 9: 100}  # the workloads' iteration caps
# Evaluations that a fit of these workloads takes on average (iterations, the
# initial one and the Fisher pass).
EVALUATIONS = {6: 10, 7: 45, 8: 47, 9: 15}
# Values of the starts of a multi-start 4D fit: below focus, in focus, above.
STARTS_4D = [(21.0, 3.5), (31.0, 3.5), (41.0, 3.5)]
OFFSET, CONVERSION = 100.0, 0.5  # camera: ADU = photons / CONVERSION + OFFSET


def listed():
    return [
        # one molecule, as an interactive tool fits the ROI under the cursor
        dict(name="fit3d_single", kind="fit", fittype=6, n=1, s=13, precision="f32"),
        # the ROIs of one or two camera frames, as an acquisition loop fits them
        dict(name="fit3d_frame", kind="fit", fittype=6, n=300, s=13, precision="f32"),
        # a file's block of ROIs through the drop-in call, host arrays in and out
        dict(name="fit3d_host", kind="host", n=20000, s=13),
        # a whole acquisition of mixed ROI sizes, resident on the device
        dict(name="fit3d_batch", kind="batch", n=1000000),
        # colour classification of an acquisition's block of ROIs
        dict(name="fit4d_block", kind="fit", fittype=7, n=40000, s=13, precision="f32"),
        # one frame's ROIs fitted from three z starts, the GUI's loop
        dict(name="fit4d_starts", kind="fit", fittype=7, n=300, s=15, precision="f32", starts=3),
        # dipole orientation of an acquisition's block of ROIs
        dict(name="fit5d_block", kind="fit", fittype=8, n=8000, s=17, precision="f32"),
        # four-channel interference ROIs
        dict(name="fit4pi_block", kind="fit", fittype=9, n=8000, s=16, precision="f32"),
        # a block refitted at the parity grade
        dict(name="fit3d_parity", kind="fit", fittype=6, n=10000, s=13, precision="parity"),
        # a sample refitted in double precision, to check a pipeline
        dict(name="fit3d_f64", kind="fit", fittype=6, n=3000, s=11, precision="f64"),
        # a chunk of camera frames to ROIs
        dict(name="frames_512", kind="frames", frames=64, height=512, width=512, emitters=150,
             s=13, sigma=1.0),
        # coefficients of the 5D orientation model
        dict(name="coeffs_5d", kind="coeffs", dims="34x34x41x18x9"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "fit", "fit", "host", "batch", "frames", "coeffs"])
    if kind == "host":
        return dict(kind="host", n=_log_int(rng, 1, 200000), s=rng.choice([7, 9, 11, 13, 15, 17, 21]))
    if kind == "batch":
        return dict(kind="batch", n=_log_int(rng, 1000, 800000))
    if kind == "frames":
        h, w = _log_int(rng, 64, 640), _log_int(rng, 64, 640)
        return dict(kind="frames", frames=_log_int(rng, 1, 64), height=h, width=w,
                    emitters=max(1, h * w // rng.randint(1200, 4000)),
                    s=rng.choice([7, 9, 11, 13, 15, 17]), sigma=rng.choice([0.8, 1.0, 1.3, 1.6]))
    if kind == "coeffs":
        d = [rng.randint(20, 40), 0, rng.randint(20, 64)]
        d[1] = d[0]
        d += [rng.randint(4, 34)] if rng.random() < 0.6 else []
        d += [rng.randint(4, 9)] if len(d) == 4 and rng.random() < 0.5 else []
        return dict(kind="coeffs", dims="x".join(map(str, d)))
    fittype, precision = rng.choice([(6, "f32"), (6, "f32"), (6, "f32"), (7, "f32"), (7, "f32"),
                                     (8, "f32"), (8, "f32"), (9, "f32"), (9, "f32"),
                                     (6, "parity"), (7, "parity"), (6, "f64")])
    most = {(6, "f32"): 200000, (7, "f32"): 60000, (8, "f32"): 12000, (9, "f32"): 40000,
            (6, "parity"): 40000, (7, "parity"): 4000, (6, "f64"): 4000}[fittype, precision]
    s = rng.choice({6: [7, 9, 11, 13, 15, 17, 21], 7: [9, 11, 13, 15, 17], 8: [13, 15, 17, 19],
                    9: [12, 14, 16]}[fittype])
    case = dict(kind="fit", fittype=fittype, n=_log_int(rng, 1, most), s=s, precision=precision)
    if precision == "f32" and fittype == 6 and rng.random() < 0.3:
        case["scmos"] = True
    if precision == "f32" and fittype == 7 and rng.random() < 0.4:
        case["starts"] = rng.choice([2, 3])
        case["n"] = max(1, case["n"] // 3)
    return case


# ---------------------------------------------------------------------------
# Inputs, drawn on the device from the seed.


class _Draw:
    def __init__(self, seed):
        self.g = torch.Generator("cuda")
        self.g.manual_seed(seed)

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, generator=self.g, device="cuda", dtype=torch.float64)

    def log_uniform(self, lo, hi, *shape):
        return torch.exp(self.uniform(math.log(lo), math.log(hi), *shape))

    def poisson(self, mean):
        return torch.poisson(mean.float(), generator=self.g)


def _pixel_gauss(center, sigma, n):
    """Pixel-integrated unit Gaussians on pixels 0 .. n-1, shape (N, n)."""
    edges = torch.arange(n + 1, device="cuda", dtype=torch.float64)[None, :] - 0.5
    u = (edges - center[:, None]) / (math.sqrt(2.0) * sigma[:, None])
    return torch.diff(0.5 * (1.0 + torch.erf(u)), dim=1)


def _astig(z_nm, sigma0):
    return (sigma0 * torch.sqrt(1.0 + ((z_nm - 200.0) / 400.0) ** 2),
            sigma0 * torch.sqrt(1.0 + ((z_nm + 200.0) / 400.0) ** 2))


def _rois(d, fittype, n, s):
    """(ROIs of fit type 6, 7 or 8): Poisson images of the model's PSF."""
    c = (s - 1) / 2.0
    spread = 1.0 if fittype == 8 else 1.5
    x, y = c + d.uniform(-spread, spread, n), c + d.uniform(-spread, spread, n)
    zr = 300.0 if fittype == 8 else 600.0
    z = d.uniform(-zr, zr, n)
    if fittype == 8:
        photons, bg = d.uniform(2000.0, 8000.0, n), d.uniform(5.0, 20.0, n)
        phi, th = d.uniform(0.0, 2 * math.pi, n), torch.deg2rad(d.uniform(10.0, 70.0, n))
        st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(phi), torch.cos(phi)
        sx, sy = _astig(z, 1.3)
        sm = 0.55 * (sx + sy)
        psf = 0.0
        for wgt, gx, gy in ((st ** 2 * cp ** 2, sx, sy), (st ** 2 * sp ** 2, sy, sx), (ct ** 2, sm, sm)):
            psf = psf + (wgt[:, None] * _pixel_gauss(x + 0.4 * st * cp, gx, s))[:, :, None] \
                * _pixel_gauss(y + 0.4 * st * sp, gy, s)[:, None, :]
    else:
        if fittype == 7:
            photons, bg = d.log_uniform(800.0, 4000.0, n), d.uniform(5.0, 15.0, n)
            sigma0 = 1.2 + 0.25 * d.uniform(0.0, 1.0, n)
        else:
            photons, bg = d.log_uniform(1000.0, 5000.0, n), d.uniform(5.0, 20.0, n)
            sigma0 = 1.3
        sx, sy = _astig(z, sigma0)
        psf = _pixel_gauss(x, sx, s)[:, :, None] * _pixel_gauss(y, sy, s)[:, None, :]
    return d.poisson(bg[:, None, None] + photons[:, None, None] * psf)


def _rois_4pi(d, n, s):
    """Four-channel ROIs (4, n, s, s), the channels' offsets and the starts."""
    c = (s - 1) / 2.0
    x, y = c + d.uniform(-1.0, 1.0, n), c + d.uniform(-1.0, 1.0, n)
    z, phi = d.uniform(-500.0, 500.0, n), d.uniform(0.0, 2 * math.pi, n)
    psi = 2 * math.pi * z / wl.PHASE_PERIOD_NM_C4 + phi
    photons, bg = d.log_uniform(500.0, 2500.0, n), d.uniform(5.0, 20.0, n)
    dT = torch.zeros((n, 4, 6), device="cuda")
    dT[:, :, :2] = d.uniform(-0.5, 0.5, n, 4, 2).float()
    sx, sy = _astig(z, 1.3)
    rois = torch.empty((4, n, s, s), device="cuda")
    for k in range(4):
        mod = photons * (1.0 + 0.8 * torch.cos(psi + 0.5 * math.pi * k))
        psf = _pixel_gauss(x + dT[:, k, 0], sx, s)[:, :, None] * _pixel_gauss(y + dT[:, k, 1], sy, s)[:, None, :]
        rois[k] = d.poisson(bg[:, None, None] + mod[:, None, None] * psf)
    z0 = torch.full((n,), float(wl.z_to_param(0.0)), device="cuda")
    return rois, dT, z0, torch.ones(n, device="cuda")


def _shifts_4pi():
    return (np.arange(4) * 0.5 * np.pi / wl.PHI_STEP_C4).astype(np.float32)


def _model(fittype, s):
    if fittype == 6:
        return bsfit.Model(6, wl.coeff3d())
    if fittype == 7:
        return bsfit.Model(7, wl.coeff4d(), init_p=np.array([31.0, 3.5], np.float32))
    if fittype == 8:
        c5, c3 = wl.coeff5d()
        ip = [wl.z_to_param(0.0, -400.0), wl.phi_to_w(np.pi), wl.theta_to_u(np.deg2rad(40.0)), 0.7]
        return bsfit.Model(8, c5, coeff3=c3, init_p=np.array(ip, np.float32))
    return bsfit.Model4Pi(wl.coeff4pi_c4(s), _shifts_4pi())


def _batch_counts(n):
    return ((11, n // 4), (13, n - 2 * (n // 4)), (17, n // 4))


def _frames(d, case):
    """Camera frames (F, W, H) in ADU: Poisson images of astigmatic emitters, one
    in each of E cells of every frame, away from the border."""
    F, H, W, E = case["frames"], case["height"], case["width"], case["emitters"]
    m, edge = F * E, case["s"]
    sx, sy = _astig(d.uniform(-300.0, 300.0, m), 1.3)
    photons = d.log_uniform(1500.0, 6000.0, m)
    cols = max(1, math.ceil(math.sqrt(E * W / H)))
    rows = math.ceil(E / cols)
    cell = torch.arange(E, device="cuda").repeat(F)
    x = edge + (cell % cols + d.uniform(0.2, 0.8, m)) * ((W - 2 * edge) / cols)
    y = edge + (cell // cols + d.uniform(0.2, 0.8, m)) * ((H - 2 * edge) / rows)
    gx = (photons[:, None] * _pixel_gauss(x, sx, W)).view(F, E, W)
    gy = _pixel_gauss(y, sy, H).view(F, E, H)
    mean = 10.0 + torch.bmm(gx.transpose(1, 2), gy)
    return d.poisson(mean) / CONVERSION + OFFSET


def _coeff_samples(d, dims):
    """A smooth stack with noise, shape the reversed dims (fastest axis last)."""
    shape = tuple(reversed(dims))
    x = torch.rand(shape, generator=d.g, device="cuda", dtype=torch.float64) * 1e-3
    envelope = torch.ones((), device="cuda", dtype=torch.float64)
    for k in shape:
        t = torch.linspace(-2.0, 2.0, k, device="cuda", dtype=torch.float64)
        envelope = envelope[..., None] * torch.exp(-t * t)
    return x + envelope


def _dims(case):
    return [int(v) for v in case["dims"].split("x")]


def prepare(case, seed):
    d = _Draw(seed)
    st = dict(case)
    if case["kind"] == "coeffs":
        st["samples"] = _coeff_samples(d, _dims(case))
    elif case["kind"] == "frames":
        st["images"] = _frames(d, case)
        st["kernel"] = bsfit.peak_kernel(1, case["sigma"])
    elif case["kind"] == "host":
        st["rois"] = _rois(d, 6, case["n"], case["s"]).cpu().numpy()
        st["coeff"] = wl.coeff3d()
    elif case["kind"] == "batch":
        m = _model(6, 13)
        st["rois"] = [_rois(d, 6, n, s) for s, n in _batch_counts(case["n"])]
        st["batch"] = bsfit.Batch([(m, r, ITERATIONS[6]) for r in st["rois"]])
    else:
        st["model"] = _model(case["fittype"], case["s"])
        if case["fittype"] == 9:
            st["rois"], st["dT"], st["z0"], st["phi0"] = _rois_4pi(d, case["n"], case["s"])
        else:
            st["rois"] = _rois(d, case["fittype"], case["n"], case["s"])
        if case.get("scmos"):
            # read-noise variance over gain^2 of an sCMOS chip, and its noise
            st["var"] = (1.0 + 4.0 * d.uniform(0.0, 1.0, *st["rois"].shape) ** 4).float()
            noise = torch.randn(st["rois"].shape, generator=d.g, device="cuda") * st["var"].sqrt()
            st["rois"] = (st["rois"] + noise).contiguous()
    return st


def run(state):
    kind = state["kind"]
    if kind == "coeffs":
        return bsfit.bsarray_coeffs_torch(state["samples"])
    if kind == "frames":
        return bsfit.find_rois_torch(state["images"], OFFSET, CONVERSION, state["kernel"], True,
                                     _cutoff(state["sigma"]), state["s"], capacity=_capacity(state))
    if kind == "host":
        return bsfit.GPUmleFit_LM_multiD(state["rois"], 6, ITERATIONS[6], state["coeff"])
    if kind == "batch":
        return state["batch"].run()
    m, rois, its = state["model"], state["rois"], ITERATIONS[state["fittype"]]
    if state["fittype"] == 9:
        return m.fit_torch(rois, its, state["z0"], state["phi0"], state["dT"])
    if state["precision"] == "f64":
        return m.fit_f64_torch(rois, its)
    if state.get("scmos"):
        return m.fit_scmos_torch(rois, state["var"], its)
    if state.get("starts"):
        return m.fit_multistart_torch(rois, its, STARTS_4D[:state["starts"]])
    return m.fit_torch(rois, its, precision=state["precision"])


def _cutoff(sigma):
    """Filter response (photons) above which a maximum is an emitter."""
    return 12.0 / sigma


def _capacity(case):
    """ROIs that the program's buffers hold for a chunk of frames: the chunk is
    sized so that they are filled."""
    return max(1, 4 * case["frames"] * case["emitters"] // 5)


def work(case):
    kind = case["kind"]
    if kind == "coeffs":
        dims = _dims(case)
        n = math.prod(dims)
        # per axis and sample: a multiply-add each way and the gain
        return {"bytes": 8 * n + 4 * math.prod(k + 2 for k in dims), "flops": 5 * len(dims) * n}
    if kind == "frames":
        px = case["frames"] * case["height"] * case["width"]
        k = max(math.ceil(6.0 * case["sigma"] + 1.0), 3)
        found = _capacity(case)
        # the kernel is a difference of two separable ones: two passes each
        return {"bytes": 4 * px + found * (4 * case["s"] ** 2 + 12), "flops": 8 * k * px}
    if kind == "batch":
        parts = [(6, s, n) for s, n in _batch_counts(case["n"])]
    elif kind == "host":
        parts = [(6, case["s"], case["n"])]
    else:
        parts = [(case["fittype"], case["s"], case["n"])]
    b = f = 0
    for ft, s, n in parts:
        ch = 4 if ft == 9 else 1
        nv = 6 if ft == 9 else bsfit.NUM_PARAMS[ft]
        out = 8 if case.get("precision") == "f64" else 4
        planes = ch * (2 if case.get("scmos") else 1)
        b += n * (4 * planes * s * s + out * (2 * nv + 2) + (104 if ft == 9 else 0))
        f += n * EVALUATIONS[ft] * case.get("starts", 1) * bsfit.eval_flops(ft, s)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# Outputs in 64 bits, from plain torch.


def _prefilter_matrix(n):
    """Sample values to mirror-boundary cubic B-spline coefficients, dense."""
    a = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for i in range(n):
        a[i, i] += 4.0 / 6.0
        for j in (i - 1, i + 1):
            j = -j if j < 0 else 2 * n - 2 - j if j >= n else j
            a[i, j] += 1.0 / 6.0
    return torch.linalg.inv(a)


def _exact_coeffs(samples):
    c = samples
    for ax in range(c.dim()):
        n = c.shape[ax]
        c = torch.movedim(torch.tensordot(_prefilter_matrix(n), c, dims=([1], [ax])), 0, ax)
        i = torch.tensor([1] + list(range(n)) + [n - 2], device="cuda")
        c = c.index_select(ax, i)
    return c


def _exact_frames(images, kernel, cutoff, s, most):
    """Conversion, filter, strict 3 x 3 maxima, border rule and cut-outs."""
    photons = (images.double() - OFFSET) * CONVERSION  # (F, W, H)
    k = kernel.shape[0]
    o = (k - 1) // 2
    # h[u, v]: u the row (y) offset, v the column (x) offset
    h = torch.as_tensor(np.asarray(kernel, np.float64).T.copy(), device="cuda")
    base = photons - photons[:, 0, :].amin(dim=1)[:, None, None]
    F, W, H = base.shape
    pad = torch.nn.functional.pad(base, (o, k - 1 - o, o, k - 1 - o))
    img = torch.zeros_like(base)
    for v in range(k):
        for u in range(k):
            img += h[v, u] * pad[:, v:v + W, u:u + H]
    dx = s // 2
    hit = torch.zeros(base.shape, dtype=torch.bool, device="cuda")
    centre = img[:, 1:-1, 1:-1]
    keep = centre > cutoff
    for a in range(3):
        for b in range(3):
            if (a, b) != (1, 1):
                keep &= centre > img[:, a:a + W - 2, b:b + H - 2]
    hit[:, 1:-1, 1:-1] = keep
    inside = torch.zeros_like(hit)
    inside[:, dx:W - dx, dx:H - dx] = True
    f, x, y = torch.nonzero(hit & inside, as_tuple=True)
    r = torch.arange(-dx, dx + 1, device="cuda")
    f, x, y = f[:most], x[:most], y[:most]
    rois = photons[f[:, None, None], (x[:, None] + r)[:, :, None], (y[:, None] + r)[:, None, :]]
    return rois, torch.stack([x + 1, y + 1, f + 1], dim=1).double()


def _knot(pos, n):
    c = torch.floor(pos).clamp(min=1).clamp(max=n - 1)
    return torch.where(pos == n, torch.full_like(c, n), c).long()


def _b3(x):
    a = x.abs()
    return torch.where(a < 1, 2.0 / 3.0 - a * a + 0.5 * a ** 3, ((2.0 - a).clamp(min=0) ** 3) / 6.0)


def _b2(x):
    a = x.abs()
    return torch.where(a < 0.5, 0.75 - a * a, 0.5 * (1.5 - a).clamp(min=0) ** 2)


def _weights(pos):
    """Value weights of nodes -1 .. 2 and derivative weights of differences
    (-1, 0), (0, 1), (1, 2) at the fractional part of pos: (N, 4), (N, 3)."""
    t = (pos - torch.floor(pos))[:, None]
    o = torch.arange(-1, 3, device="cuda", dtype=torch.float64)
    return _b3(t - o), _b2(t - (o[:3] + 0.5))


def _psf(coeff, th, s):
    """Value and d/dX, d/dY, d/dZ (and d/dW of a 4D model) of the spline at every
    pixel (N, s, s), for th = (x, y, z[, w]) each (N,)."""
    D = coeff.dim()
    n = [k - 3 for k in reversed(coeff.shape)]
    N = th[0].shape[0]
    off = (n[1] - s) / 2.0
    j = torch.arange(s, device="cuda", dtype=torch.float64)
    xc, yc = (s + 1) // 2 - th[0], (s + 1) // 2 - th[1]
    kx, ky = _knot(xc[:, None] + j + off, n[1]), _knot(yc[:, None] + j + off, n[0])
    xb, yb = kx.amin(1, keepdim=True) - 1, ky.amin(1, keepdim=True) - 1
    a = torch.arange(s + 4, device="cuda")
    xn, yn = (xb + a).clamp(max=coeff.shape[-2] - 1), (yb + a).clamp(max=coeff.shape[-1] - 1)
    k4 = torch.arange(-1, 3, device="cuda")
    iz = (_knot(th[2], n[2])[:, None] + k4)
    bz, dz = _weights(th[2])
    if D == 4:
        iw = (_knot(th[3], n[3])[:, None] + k4)
        bw, dw = _weights(th[3])
        c = coeff[iw[:, :, None, None, None], iz[:, None, :, None, None], xn[:, None, None, :, None],
                  yn[:, None, None, None, :]]
        v = torch.einsum("nwzxy,nz->nwxy", c, bz)
        d = torch.einsum("nwzxy,nz->nwxy", c[:, :, 1:] - c[:, :, :-1], dz)
        maps = [torch.einsum("nwxy,nw->nxy", v, bw), torch.einsum("nwxy,nw->nxy", d, bw),
                torch.einsum("nwxy,nw->nxy", v[:, 1:] - v[:, :-1], dw)]
    else:
        c = coeff[iz[:, :, None, None], xn[:, None, :, None], yn[:, None, None, :]]
        maps = [torch.einsum("nzxy,nz->nxy", c, bz),
                torch.einsum("nzxy,nz->nxy", c[:, 1:] - c[:, :-1], dz)]
    bx, dx = _weights(xc)
    by, dy = _weights(yc)
    gx = (kx - 1 - xb)[:, :, None] + torch.arange(4, device="cuda")
    gy = (ky - 1 - yb)[:, :, None] + torch.arange(4, device="cuda")
    rows = torch.arange(N, device="cuda")[:, None, None]

    def along_y(m):
        return m.transpose(1, 2)[rows, gy].permute(0, 3, 1, 2)  # (N, X nodes, py, 4)

    def along_x(g):
        return g[rows, gx]  # (N, px, 4, py)

    q = along_y(maps[0])
    val = along_x(torch.einsum("nxpk,nk->nxp", q, by))
    gdy = along_x(torch.einsum("nxpk,nk->nxp", q[..., 1:] - q[..., :-1], dy))
    out = [torch.einsum("npkq,nk->npq", val, bx),
           torch.einsum("npkq,nk->npq", val[:, :, 1:] - val[:, :, :-1], dx),
           torch.einsum("npkq,nk->npq", gdy, bx)]
    for m in maps[1:]:
        out.append(torch.einsum("npkq,nk->npq", along_x(torch.einsum("nxpk,nk->nxp", along_y(m), by)), bx))
    return out


class _Exact:
    """The LM fit of fit type 6 and of the 4Pi model, in 64 bits."""

    def __init__(self, coeff, rois, var=None, dT=None, shifts=None):
        self.coeff, self.rois, self.var, self.dT, self.shifts = coeff, rois, var, dT, shifts
        self.s = rois.shape[-1]
        self.pi4 = rois.dim() == 4
        self.nv = 6 if self.pi4 else 5
        self.n = [k - 3 for k in reversed(coeff.shape)]

    def wrap(self, w):
        p = self.n[3] - 1
        return torch.where(w < 1, w + p, torch.where(w >= self.n[3], w - p, w))

    def sums(self, at, th, fisher):
        """Deviance or log-likelihood, gradient, Hessian or Fisher matrix of the
        ROIs `at` at th (N, nv)."""
        total = [0.0, 0.0, 0.0]
        for ch in range(4 if self.pi4 else 1):
            t = th
            if self.pi4:
                t = th + self.dT[at, ch]
                t = torch.cat([t[:, :5], self.wrap(t[:, 5] + self.shifts[ch])[:, None]], dim=1)
            pos = [t[:, 0], t[:, 1]] + [t[:, k] for k in range(4, self.nv)]
            f, dx, dy, *rest = _psf(self.coeff, pos, self.s)
            N = t[:, 2, None, None]
            model = t[:, 3, None, None] + N * f
            du = torch.stack([-N * dx, -N * dy, f, torch.ones_like(f)] + [N * r for r in rest], dim=1).flatten(2)
            data = (self.rois[ch] if self.pi4 else self.rois)[at]
            if self.var is not None:
                model, data = model + self.var[at], data + self.var[at]
            model, data = model.flatten(1), data.flatten(1)
            seen = data > 0
            d1 = torch.where(seen, data, torch.ones_like(data))
            if fisher:
                m1 = torch.where(model > 0, model, torch.ones_like(model))
                e = torch.where(seen, d1 * torch.log(m1) - model - d1 * torch.log(d1) + d1, -model)
                e = torch.where(model > 0, e, torch.zeros_like(e))
                w, t1 = 1.0 / model, torch.zeros_like(model)
            else:
                e = 2.0 * torch.where(seen, (model - d1) + d1 * torch.log(d1 / model), model)
                dm = torch.where(seen, data / model, torch.zeros_like(data))
                w, t1 = dm / model, 1.0 - dm
            total[0] = total[0] + e.sum(1)
            total[1] = total[1] + torch.einsum("np,nkp->nk", t1, du)
            total[2] = total[2] + torch.einsum("np,nkp,nlp->nkl", w, du, du)
        return total

    def start(self, z0, w0):
        s = self.s
        planes = self.rois if self.pi4 else self.rois[None]
        j = torch.arange(s, device="cuda", dtype=torch.float64)
        guess = 0.0
        for ch, r in enumerate(planes):
            t = r.sum((1, 2))
            hi, lo = r.amax((1, 2)).clamp(min=0), r.amin((1, 2))
            g = torch.stack([torch.einsum("nxy,y->n", r, j) / t, torch.einsum("nxy,x->n", r, j) / t,
                             ((hi - lo) * 2 * float(np.float32(3.141592)) * 2.25).clamp(min=0),
                             lo.clamp(min=0.01)], dim=1)
            if self.pi4:
                g[:, :2] -= self.dT[:, ch, :2]
            guess = guess + g
        rest = [z0] + ([self.wrap(w0)] if self.pi4 else [])
        return torch.cat([guess / len(planes)] + [r[:, None] for r in rest], dim=1)

    def bounds(self, p):
        top = self.n[2] - (0.5 if self.pi4 else 4)
        cols = [p[:, 0], p[:, 1], p[:, 2].clamp(min=1.0), p[:, 3].clamp(min=0.01), p[:, 4].clamp(0.0, top)]
        return torch.stack(cols + ([self.wrap(p[:, 5])] if self.pi4 else []), dim=1)

    def chunk(self, at, p, iterations):
        N, nv = p.shape
        one = torch.ones(N, device="cuda", dtype=torch.float64)
        cmax = torch.tensor([1.0, 1.0, 1e4, 20.0, 2.0, 2.0] if self.pi4 else [2.0, 2.0, 1e4, 20.0, 20.0],
                            device="cuda", dtype=torch.float64).expand(N, nv)
        st = dict(p=p, op=p, c=cmax, oc=cmax, g=0 * p, og=0 * p, lam=one, olam=one, oerr=1e13 * one)
        st["err"], st["jac"], st["hes"] = self.sums(at, p, False)
        final, count = p.clone(), torch.zeros(N, device="cuda", dtype=torch.float64)
        live = torch.arange(N, device="cuda")
        for k in range(iterations + 1):
            stop = ((st["err"] - st["oerr"]) / st["err"]).abs() < 1e-6
            stop |= k == iterations
            final[live[stop]], count[live[stop]] = st["p"][stop], float(k)
            go = ~stop
            live, st = live[go], {n: v[go] for n, v in st.items()}
            if not live.numel():
                break
            bad = st["err"] > 1.5 * st["oerr"]
            better = ~bad & (st["err"] < st["oerr"])
            for a, b in (("g", "og"), ("c", "oc"), ("p", "op")):
                st[a] = torch.where(bad[:, None], st[b], st[a])
            lam = torch.where(bad, 10.0 * st["olam"], st["lam"])
            lam = torch.where(better & (lam > 1), 0.8 * lam, torch.where(better & (lam < 1), torch.ones_like(lam), lam))
            err = torch.where(bad, st["oerr"], st["err"])
            hes = st["hes"] + torch.diag_embed((lam[:, None] - 1.0) * torch.diagonal(st["hes"], dim1=1, dim2=2))
            held = torch.diagonal(hes, dim1=1, dim2=2) == 0
            a = torch.where(held[:, :, None] | held[:, None, :], torch.zeros_like(hes), hes) + torch.diag_embed(held.double())
            low, info = torch.linalg.cholesky_ex(a)
            ok = info == 0
            rhs = torch.where(held, torch.zeros_like(st["jac"]), st["jac"])
            u = torch.cholesky_solve(rhs[:, :, None], torch.where(ok[:, None, None], low, torch.eye(nv, device="cuda", dtype=torch.float64)))[:, :, 0]
            turned = ((st["g"] == 1) & (u < 0)) | ((st["g"] == -1) & (u > 0))
            c = torch.where(turned, 0.5 * st["c"], st["c"])
            q = self.bounds(st["p"] - u / (1.0 + (u / c).abs()))
            e2, j2, h2 = self.sums(at[live], q, False)
            o, o2, o3 = ok, ok[:, None], ok[:, None, None]
            st = dict(p=torch.where(o2, q, st["p"]), op=torch.where(o2, st["p"], st["op"]),
                      c=torch.where(o2, c, st["c"]), oc=torch.where(o2, st["c"], st["oc"]),
                      g=torch.where(o2, torch.where(u > 0, 1.0, -1.0).double(), st["g"]),
                      og=torch.where(o2, st["g"], st["og"]),
                      lam=torch.where(o, lam, 10.0 * lam), olam=torch.where(o, lam, st["olam"]),
                      err=torch.where(o, e2, err), oerr=torch.where(o, err, st["oerr"]),
                      jac=torch.where(o2, j2, st["jac"]), hes=torch.where(o3, h2, hes))
        ll, _, m = self.sums(at, final, True)
        # a parameter without any derivative (z on a boundary knot): infinite variance
        held = torch.diagonal(m, dim1=1, dim2=2) == 0
        m = torch.where(held[:, :, None] | held[:, None, :], torch.zeros_like(m), m) + torch.diag_embed(held.double())
        crlb = torch.diagonal(torch.linalg.inv(m), dim1=1, dim2=2)
        crlb = torch.where(held, torch.full_like(crlb, math.inf), crlb)
        return torch.cat([final, count[:, None]], dim=1), crlb, ll

    def fit(self, iterations, z0, w0=None):
        N = z0.shape[0]
        p = self.start(z0, w0)
        size = 1000 if self.pi4 else 5000
        parts = [self.chunk(torch.arange(b, min(b + size, N), device="cuda"), p[b:b + size], iterations)
                 for b in range(0, N, size)]
        return tuple(torch.cat(v) for v in zip(*parts))


def exact(case, seed):
    """None for the fits of fit types 7 and 8: fit type 7's first Hessian is
    singular, so its first step is a ratio of rounding residuals, and both end
    in different places in two correct 64-bit builds of the method (23% and 3%
    of the ROIs). None for the double-precision fit, which follows the
    reference's order of operations: where z reaches a boundary knot, whose
    derivative is zero but for rounding, so does its step. None where it would
    take too long."""
    kind = case["kind"]
    if kind == "fit" and (case["fittype"] in (7, 8) or case["precision"] == "f64"):
        return None
    if kind == "batch" or case.get("n", 0) > 40000:
        return None
    st = prepare(case, seed)
    if kind == "coeffs":
        return _exact_coeffs(st["samples"])
    if kind == "frames":
        return _exact_frames(st["images"], st["kernel"], _cutoff(case["sigma"]), case["s"], _capacity(case))
    s = case["s"]
    if kind == "fit" and case["fittype"] == 9:
        coeff = torch.as_tensor(wl.coeff4pi_c4(s), device="cuda").double()
        e = _Exact(coeff, st["rois"].double(), dT=st["dT"].double(), shifts=[float(v) for v in _shifts_4pi()])
        out = e.fit(ITERATIONS[9], st["z0"].double(), st["phi0"].double())
        return out[0].T, out[1].T, out[2]
    coeff = torch.as_tensor(wl.coeff3d(), device="cuda").double()
    rois = torch.as_tensor(st["rois"], device="cuda").double()
    var = st["var"].double() if "var" in st else None
    z0 = torch.full((case["n"],), (coeff.shape[0] - 3) / 2.0, device="cuda", dtype=torch.float64)
    P, C, L = _Exact(coeff, rois, var=var).fit(ITERATIONS[6], z0)
    if kind == "host":
        return P, C, L
    return P.T, C.T, L
