"""The workloads by which this framework's speed is followed: what a user has it draw.

Each case goes through the public entry points -- drawImage, draw_batch, the autograd models,
StampBatch.addNoise -- from host parameters (or, for fits, device parameters) to stamps on the
device.  Sizes and distributions are those of the repository's own benchmark: catalog galaxies
(Sersic through a Kolmogorov PSF, or through a PSF image), bulge + disk galaxies through Moffat
PSFs, shape fits, large diffraction-limited stamps, chromatic galaxies, and CCD noise.

exact() evaluates the same draws in 64 bits with plain torch: closed-form profile transforms, the
Sersic and Kolmogorov Hankel integrals by a trapezoid rule on a rotated contour, GalSim's sizing
rules, a full-grid inverse FFT, and torch's own autograd for the gradients.
"""
import math
import types

import numpy as np
import torch

import galsim_b200 as galsim
from galsim_b200 import autodiff
from galsim_b200.batch import StampBatch

SCALE = 0.2          # arcsec per pixel
LARGE_SCALE = 0.05   # for the diffraction-limited stamps


def listed():
    return [
        # one object drawn by drawImage into a 64 x 64 double image: the interactive call and
        # the inner step of any program that draws object by object
        dict(name="single_64", kind="single", nx=64, ny=64),
        # a catalog exposure: 4096 galaxies, each with its own Sersic index, automatic sizes
        dict(name="catalog_4096", kind="catalog", stamps=4096, nx=0, ny=0, precision="fp32"),
        # a postage-stamp catalog in double precision, odd sizes, a batch that is no round number
        dict(name="catalog_113_fp64", kind="catalog", stamps=113, nx=53, ny=47, precision="fp64"),
        # galaxies through one PSF image (a PSF model's output), fixed stamps
        dict(name="image_psf_1024", kind="image_psf", stamps=1024, nx=48, ny=48),
        # one gradient step of a shape fit over a batch: forward, chi^2 and gradients
        dict(name="fit_1024", kind="fit", stamps=1024, nx=48, ny=48, precision="fp32"),
        # the same for a handful of objects with odd stamps in double precision, where latency counts
        dict(name="fit_29_fp64", kind="fit", stamps=29, nx=41, ny=33, precision="fp64"),
        # bulge + disk simulation, 16384 galaxies of very uneven FFT sizes
        dict(name="bulge_disk_16384", kind="bulge_disk", stamps=16384),
        # gradients of bulge + disk records (flux, Jacobian, size, n of both components)
        dict(name="bulge_disk_grad_2048", kind="bulge_disk_grad", stamps=2048, nx=64, ny=64),
        # large diffraction-limited stamps (FFTs of several thousand), single and double precision
        dict(name="large_6", kind="large", stamps=6, precision="fp32"),
        dict(name="large_2_fp64", kind="large", stamps=2, precision="fp64"),
        # CCD noise on stamps already on the device, one random stream per stamp
        dict(name="ccd_noise_1024", kind="ccd_noise", stamps=1024, nx=61, ny=57),
        # chromatic galaxies: two SEDs through an atmospheric PSF and a bandpass
        dict(name="chromatic_1024", kind="chromatic", stamps=1024, nx=32, ny=32),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["single", "catalog", "catalog", "image_psf", "fit", "fit", "bulge_disk",
                       "bulge_disk_grad", "large", "ccd_noise", "chromatic"])
    c = dict(kind=kind)
    if kind == "single":
        c.update(nx=rng.randint(24, 160), ny=rng.randint(24, 160))
    elif kind == "catalog":
        fixed = rng.random() < 0.5
        c.update(stamps=_log_int(rng, 16, 4096), nx=rng.randint(20, 96) if fixed else 0, ny=0,
                 precision=rng.choice(["fp32", "fp32", "fp64"]))
        if fixed:
            c["ny"] = rng.randint(20, 96)
    elif kind == "image_psf":
        c.update(stamps=_log_int(rng, 16, 2048), nx=rng.randint(20, 96), ny=rng.randint(20, 96))
    elif kind == "fit":
        c.update(stamps=_log_int(rng, 8, 1024), nx=rng.randint(24, 72), ny=rng.randint(24, 72),
                 precision=rng.choice(["fp32", "fp32", "fp64"]))
    elif kind == "bulge_disk":
        c.update(stamps=_log_int(rng, 64, 16384))
    elif kind == "bulge_disk_grad":
        c.update(stamps=_log_int(rng, 32, 2048), nx=rng.randint(24, 80), ny=rng.randint(24, 80))
    elif kind == "large":
        fp64 = rng.random() < 0.4
        c.update(stamps=rng.randint(1, 2 if fp64 else 6), precision="fp64" if fp64 else "fp32")
    elif kind == "ccd_noise":
        c.update(stamps=_log_int(rng, 16, 2048), nx=rng.randint(20, 96), ny=rng.randint(20, 96))
    else:
        c.update(stamps=_log_int(rng, 16, 2048), nx=rng.randint(20, 64), ny=rng.randint(20, 64))
    # sizes that differ in every draw, also where few numbers describe the case
    c["scale_of_flux"] = round(rng.uniform(0.5, 2.0), 6)
    return c


# ---- parameters --------------------------------------------------------------------------------
def _shears(rng, B, sigma, gmax):
    g = rng.normal(0., sigma, (B, 2))
    a = np.hypot(g[:, 0], g[:, 1])
    return g * np.where(a >= gmax, 0.999 * gmax / np.maximum(a, 1e-300), 1.)[:, None]


def _params(case, seed):
    """The physical parameters of a case, from the seed alone (numpy, float64)."""
    rng = np.random.default_rng([int(seed) & 0x7fffffff, 77])
    kind, B = case["kind"], int(case.get("stamps", 1))
    f0 = 1e4 * float(case.get("scale_of_flux", 1.))
    p = types.SimpleNamespace(B=B)
    auto = kind in ("bulge_disk", "large") or kind == "catalog" and not case["nx"]
    # Automatic stamp sizes follow from the shapes: there the shapes (but not the fluxes and the
    # position angles) are one population, in another order for each seed, so that the pixels
    # of all stamps together are as many for every seed.
    order, shapes = (rng.permutation(B), np.random.default_rng([B, 78])) if auto else (slice(None), rng)

    def sheared(sigma, gmax):
        g = _shears(shapes, B, sigma, gmax)[order]
        if not auto:
            return g
        t, a = rng.uniform(0., 2. * math.pi, B), np.hypot(g[:, 0], g[:, 1])
        return np.stack([a * np.cos(t), a * np.sin(t)], -1)

    if kind == "single":
        p.flux = f0 * math.exp(rng.normal(0., 0.5))
        p.hlr = math.exp(0.3 * rng.normal())
        p.g = _shears(rng, 1, 0.1, 0.6)[0]
        p.shift = rng.normal(0., 0.1, 2)
        p.fwhm = rng.uniform(0.6, 0.9)
    elif kind in ("catalog", "image_psf"):
        p.n = shapes.uniform(0.5, 4.0, B)[order]
        p.hlr = 0.5 * np.exp(0.3 * shapes.normal(size=B))[order]
        p.flux = f0 * np.exp(rng.normal(size=B))
        p.g = sheared(0.2, 0.7)
        p.fwhm = shapes.uniform(0.6, 0.9, B)[order]
        # a model PSF image: an elliptical Moffat core, 32 x 32 pixels, unit flux
        y, x = np.mgrid[:32, :32] - 15.5
        a = rng.uniform(-0.1, 0.1)
        r2 = ((1. + a) * x * x + (1. - a) * y * y) / rng.uniform(1.8, 2.4) ** 2
        im = (1. + r2) ** -3.
        p.psf_image = im / im.sum()
    elif kind == "fit":
        true = np.stack([f0 * np.exp(rng.normal(0., 0.5, B)), rng.uniform(0.3, 1.2, B), rng.uniform(1., 3., B),
                         rng.normal(0., 0.1, B), rng.normal(0., 0.1, B), rng.normal(0., 0.1, B),
                         rng.normal(0., 0.1, B)], -1)
        pert = true * (1. + rng.normal(0., 0.03, true.shape)) + \
            rng.normal(0., 0.02, true.shape) * np.array([0., 0., 0., 1., 1., 1., 1.])
        pert[:, 2] = np.clip(pert[:, 2], 0.9, 3.5)
        dt = np.float32 if case["precision"] == "fp32" else np.float64
        p.true, p.pert = true, pert.astype(dt)
        p.noise = rng.standard_normal((B, case["ny"], case["nx"]))
    elif kind in ("bulge_disk", "bulge_disk_grad", "chromatic"):
        p.flux = f0 * np.exp(rng.normal(0., 0.5, B))
        p.bf = rng.uniform(0., 0.6, B)
        p.bh = 0.4 * np.exp(shapes.normal(0., 0.3, B))[order]
        p.dh = 0.8 * np.exp(shapes.normal(0., 0.3, B))[order]
        p.g_b, p.g_d = sheared(0.2, 0.6), sheared(0.2, 0.6)
        p.beta = shapes.uniform(2.5, 4.5, B)[order]
        p.fwhm = shapes.uniform(0.5, 1.0, B)[order]
        if kind == "bulge_disk_grad":
            p.cot = rng.standard_normal((B, case["ny"], case["nx"])).astype(np.float32)
    elif kind == "large":
        p.n = shapes.uniform(4., 6., B)[order]
        p.hlr = shapes.uniform(2., 5., B)[order]
        p.flux = 10. * f0 * np.exp(rng.normal(0., 0.5, B))
    elif kind == "ccd_noise":
        p.seeds = rng.integers(1, 1 << 30, B)
        p.sky = rng.uniform(80., 120.)
    return p


# ---- the framework's side ----------------------------------------------------------------------
def _bulge_disk(p, gsp):
    bulge = galsim.Sersic(n=4., half_light_radius=p.bh, flux=p.flux * p.bf, gsparams=gsp) \
        .shear(g1=p.g_b[:, 0], g2=p.g_b[:, 1])
    disk = galsim.Exponential(half_light_radius=p.dh, flux=p.flux * (1. - p.bf), gsparams=gsp) \
        .shear(g1=p.g_d[:, 0], g2=p.g_d[:, 1])
    psf = galsim.Moffat(beta=p.beta, fwhm=p.fwhm, gsparams=gsp)
    return galsim.Convolve(galsim.Add(bulge, disk), psf, galsim.Pixel(SCALE, gsparams=gsp))


_SED_WAVES = [300., 400., 500., 600., 700., 800., 900., 1100.]
_SED_BULGE = [0.3, 0.6, 1.0, 1.4, 1.6, 1.7, 1.7, 1.6]
_SED_DISK = [2.0, 1.8, 1.4, 1.1, 0.9, 0.8, 0.7, 0.6]
_BAND = ([400., 420., 440., 460., 480., 500., 520., 540., 560., 580., 600.],
         [0.0, 0.35, 0.62, 0.71, 0.74, 0.76, 0.75, 0.70, 0.52, 0.2, 0.0])


def _chromatic(p):
    sb = galsim.SED(galsim.LookupTable(_SED_WAVES, _SED_BULGE, interpolant='linear'), 'nm', 'fphotons')
    sd = galsim.SED(galsim.LookupTable(_SED_WAVES, _SED_DISK, interpolant='linear'), 'nm', 'fphotons')
    bulge = galsim.Sersic(n=4., half_light_radius=p.bh, flux=p.flux * p.bf * 1e-2) \
        .shear(g1=p.g_b[:, 0], g2=p.g_b[:, 1]) * sb
    disk = galsim.Exponential(half_light_radius=p.dh, flux=p.flux * (1. - p.bf) * 1e-2) \
        .shear(g1=p.g_d[:, 0], g2=p.g_d[:, 1]) * sd
    psf = galsim.ChromaticAtmosphere(galsim.Kolmogorov(fwhm=0.7), 500., zenith_angle=30. * galsim.degrees,
                                     parallactic_angle=20. * galsim.degrees)
    bp = galsim.Bandpass(galsim.LookupTable(*_BAND, interpolant='linear'), 'nm')
    return galsim.Convolve(galsim.Add(bulge, disk), psf), bp


def _target(case, p, dev):
    """A fit's data: the model at the true parameters plus noise at SNR 50, and its 1 / sigma
    (float32 images, as read from a survey's files)."""
    img = _fit_images(torch.as_tensor(p.true, device=dev), case, dev)
    sigma = torch.sqrt((img ** 2).sum((1, 2))) / 50.
    target = img + sigma[:, None, None] * torch.as_tensor(p.noise, device=dev)
    return target.float(), (1. / sigma).float()[:, None, None]


def prepare(case, seed):
    dev = torch.device("cuda")
    p, kind = _params(case, seed), case["kind"]
    s = types.SimpleNamespace(case=case, kind=kind, p=p)
    if kind == "single":
        s.image = galsim.ImageD(case["nx"], case["ny"])
    elif kind == "catalog":
        gal = galsim.Sersic(n=p.n, half_light_radius=p.hlr, flux=p.flux).shear(g1=p.g[:, 0], g2=p.g[:, 1])
        s.obj = galsim.Convolve(gal, galsim.Kolmogorov(fwhm=p.fwhm), galsim.Pixel(SCALE))
    elif kind == "image_psf":
        psf = galsim.InterpolatedImage(galsim.Image(p.psf_image, scale=SCALE))
        gal = galsim.Sersic(n=p.n, half_light_radius=p.hlr, flux=p.flux).shear(g1=p.g[:, 0], g2=p.g[:, 1])
        s.obj = galsim.Convolve(gal, psf)
    elif kind == "fit":
        psf = galsim.Convolve(galsim.Moffat(beta=2.5, fwhm=0.8), galsim.Pixel(SCALE))
        fp32 = case["precision"] == "fp32"
        s.model = autodiff.GalaxyModel(psf, case["nx"], case["ny"], SCALE, precision=case["precision"],
                                       dtype=np.float32 if fp32 else np.float64)
        s.target, s.isig = _target(case, p, dev)
        s.params = torch.as_tensor(p.pert, device=dev)
    elif kind == "bulge_disk":
        s.obj = _bulge_disk(p, galsim.GSParams(minimum_fft_size=32))
    elif kind == "bulge_disk_grad":
        s.plan = autodiff.RecordPlan(_bulge_disk(p, galsim.GSParams(minimum_fft_size=32)), case["nx"], case["ny"], SCALE)
        s.plan.want = 0b11                  # the bulge and the disk
        rec = s.plan.records()
        s.records = {k: v.float() if k.startswith("leaf_") else v for k, v in rec.items()}
        s.cot = torch.as_tensor(p.cot, device=dev)
    elif kind == "large":
        s.obj = galsim.Convolve(galsim.Sersic(n=p.n, half_light_radius=p.hlr, flux=p.flux),
                                galsim.Airy(lam_over_diam=0.1, obscuration=0.3), galsim.Pixel(LARGE_SCALE))
    elif kind == "ccd_noise":
        nx, ny, B = case["nx"], case["ny"], p.B
        g = torch.Generator(device=dev)
        g.manual_seed(int(seed) & 0x7fffffff)
        flux = 1e4 * float(case.get("scale_of_flux", 1.)) * torch.exp(torch.randn(B, 1, 1, device=dev, generator=g))
        w = 2. * (2. + 3. * torch.rand(B, 1, 1, device=dev, generator=g)) ** 2
        x = torch.arange(nx, device=dev)[None, None, :] - (nx - 1) / 2.
        y = torch.arange(ny, device=dev)[None, :, None] - (ny - 1) / 2.
        s.clean = (flux / (math.pi * w) * torch.exp(-(x * x + y * y) / w)).float().reshape(-1)
        s.nx, s.ny = np.full(B, nx, np.int64), np.full(B, ny, np.int64)
        s.offsets = np.arange(B, dtype=np.int64) * (nx * ny)
        s.noise = galsim.CCDNoise(sky_level=p.sky, gain=1.5, read_noise=5.)
    else:
        s.obj, s.bandpass = _chromatic(p)
    return s


def _stamps(sb, fp64=False):
    out = dict(pixels=sb.flat, nx=sb.nx, ny=sb.ny)
    if fp64:
        out["added_flux"] = sb.added_flux
    return out


def run(s):
    case, p, kind = s.case, s.p, s.kind
    size = dict(nx=case["nx"], ny=case["ny"]) if case.get("nx") else {}
    if kind == "single":
        # one object at a time is made and drawn in one go
        gal = galsim.Exponential(flux=p.flux, half_light_radius=p.hlr).shear(g1=p.g[0], g2=p.g[1]) \
            .shift(p.shift[0], p.shift[1])
        obj = galsim.Convolve(gal, galsim.Moffat(beta=3.0, fwhm=p.fwhm), galsim.Pixel(SCALE))
        im = obj.drawImage(s.image, scale=SCALE, method='fft')
        return dict(pixels=im.array)
    if kind == "catalog":
        fp64 = case["precision"] == "fp64"
        return _stamps(galsim.draw_batch(s.obj, scale=SCALE, dtype=np.float64 if fp64 else np.float32,
                                         precision=case["precision"], **size), fp64)
    if kind == "image_psf":
        return _stamps(galsim.draw_batch(s.obj, scale=SCALE, method='no_pixel', **size))
    if kind == "fit":
        q = s.params.detach().requires_grad_(True)
        img = s.model(q)
        chi2 = (((img - s.target) * s.isig) ** 2).sum()
        chi2.backward()
        return dict(image=img.detach(), grad=q.grad)
    if kind == "bulge_disk":
        return _stamps(galsim.draw_batch(s.obj, scale=SCALE))
    if kind == "bulge_disk_grad":
        rec = {k: v.detach().requires_grad_(k.startswith("leaf_")) for k, v in s.records.items()}
        img = autodiff.draw_records(s.plan, **rec)
        img.backward(s.cot)
        return dict(image=img.detach(), **{k: rec[k].grad for k in rec if k.startswith("leaf_")})
    if kind == "large":
        fp64 = case["precision"] == "fp64"
        return _stamps(galsim.draw_batch(s.obj, scale=LARGE_SCALE, dtype=np.float64 if fp64 else np.float32,
                                         precision=case["precision"]), fp64)
    if kind == "ccd_noise":
        sb = StampBatch(s.clean.clone(), s.offsets, s.nx, s.ny, None, None, None, None, None, np.float32, SCALE, None)
        return dict(draws=sb.addNoise(s.noise, p.seeds), pixels=sb.flat)
    return _stamps(galsim.draw_batch(s.obj, scale=SCALE, bandpass=s.bandpass, **size))


# ---- the same draws in 64 bits ------------------------------------------------------------------
_FOLD, _MAXK, _KACC, _XACC, _MIN_HLR = 5e-3, 1e-3, 1e-5, 1e-5, 5.


def _contour(dev):
    """Nodes and weights of int_0^inf r J0(k r) f(r) dr = k^-2 Re sum_j W_j f(s_j e^{i phi} / k), the
    contour turned by phi = pi / 8 into the half plane where the Hankel function decays."""
    phi, h = math.pi / 8., 0.07
    u = torch.arange(-40., 4.7, h, dtype=torch.float64, device=dev)
    s = torch.exp(u)
    a = phi - math.pi / 2.                        # H0(1)(z) = 2 / (pi i) K0(-i z)
    t = torch.arange(0., 8., 0.02, dtype=torch.float64, device=dev)
    ch = torch.cosh(t)
    ex = s[:, None] * ch
    e = torch.exp(-ex * math.cos(a))
    w = torch.ones_like(t)
    w[0] = 0.5
    w = w * 0.02
    # the tail beyond the t grid matters only where s is tiny; there K0(z) = -ln(z / 2) - gamma
    kr = (w * e * torch.cos(ex * math.sin(a))).sum(1)
    ki = -(w * e * torch.sin(ex * math.sin(a))).sum(1)
    small = s < 0.05
    z2 = s * s / 4.
    q = torch.complex(torch.cos(torch.full_like(s, 2. * a)) * z2, torch.sin(torch.full_like(s, 2. * a)) * z2)
    ln = torch.complex(torch.log(s / 2.) + 0.5772156649015329, torch.full_like(s, a))
    k0 = -ln * (1 + q + q * q / 4. + q ** 3 / 36.) + q + q * q * 0.375 + q ** 3 * (11. / 216.)
    K = torch.where(small, k0, torch.complex(kr, ki))
    W = s * s * h * complex(math.cos(2. * phi), math.sin(2. * phi)) * K * complex(0., -2. / math.pi)
    return u, W.real.contiguous(), W.imag.contiguous(), phi


def _hankel(lnk, n, con):
    """k^2 times the order-0 Hankel transform of exp(-r^(1/n)) at ln k (n broadcast against lnk)."""
    u, wr, wi, phi = con
    x = torch.exp((u - lnk[..., None]) / n[..., None])
    c, s = torch.cos(phi / n)[..., None], torch.sin(phi / n)[..., None]
    e = torch.exp(-x * c)
    return (e * (wr * torch.cos(x * s) + wi * torch.sin(x * s))).sum(-1)


def _sersic_ft(ksq, n, con):
    """The unit-flux transform at ksq = (k r0)^2."""
    norm = n * torch.exp(torch.special.gammaln(2. * n))
    tiny = ksq < 1e-24
    safe = torch.where(tiny, torch.ones_like(ksq), ksq)
    v = _hankel(0.5 * torch.log(safe), n.expand_as(safe), con) / safe / norm
    return torch.where(tiny, torch.ones_like(v), v)


def _sersic_b(n):
    """b(n) with P(2n, b) = 1/2, differentiable through dP/dn and dP/db."""
    a = 2. * n.detach()
    b = 2. * n.detach() - 1. / 3.
    lo, hi = torch.zeros_like(b), 4. * b + 4.
    half = torch.full_like(b, 0.5)
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        up = torch.special.gammainc(a, mid) < half
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    b = 0.5 * (lo + hi)
    if not n.requires_grad:
        return b
    # dP/da = int_0^b t^(a-1) e^-t ln t dt / Gamma(a) - psi(a) P, by a trapezoid rule in ln t
    v = torch.arange(-80., 0., 0.002, dtype=torch.float64, device=n.device)
    w = torch.full_like(v, 0.002)
    lt = torch.log(b)[:, None] + v
    f = torch.exp(a[:, None] * lt - torch.exp(lt) - torch.special.gammaln(a)[:, None]) * lt
    end = torch.exp(a * torch.log(b) - b - torch.special.gammaln(a)) * torch.log(b)
    # the end term's half weight, and its Euler-Maclaurin correction h^2 / 12 f'
    d = torch.exp(a * torch.log(b) - b - torch.special.gammaln(a)) * (1. + torch.log(b) * (a - b))
    dpa = (f * w).sum(1) + 0.5 * 0.002 * end - 0.002 ** 2 / 12. * d - torch.special.digamma(a) * 0.5
    dpb = torch.exp((a - 1.) * torch.log(b) - b - torch.special.gammaln(a))
    return b - (2. * dpa / dpb) * (n - n.detach())


def _moffat_ft(k, beta):
    """The unit-flux transform at k rD, K_nu by the trapezoid rule on its cosh integral."""
    nu = beta - 1.
    x = torch.clamp(k, min=1e-9)
    t = torch.arange(0., 26., 0.1, dtype=torch.float64, device=k.device)
    ln = (1. - nu) * math.log(2.) - torch.special.gammaln(nu) + nu * torch.log(x)
    out = torch.zeros_like(x)
    for j, tj in enumerate(t.tolist()):
        term = torch.exp(ln - x * math.cosh(tj) + nu * tj) * 0.5 * (1. + torch.exp(-2. * nu * tj))
        out = out + (0.05 if j == 0 else 0.1) * term
    return torch.where(k < 1e-9, torch.ones_like(out), out)


def _airy_ft(k, lod, obs):
    """The unit-flux transform of an obscured Airy disc: its pupil's autocorrelation."""
    t = k * lod / math.pi
    d = t                                          # pupil radius 1, separation d

    def lens(r, s):
        area = torch.zeros_like(d)
        inner = d <= abs(r - s)
        both = (d < r + s) & ~inner
        dd = torch.where(both, d, torch.full_like(d, abs(r - s) + 0.5 * min(r, s)))
        ar = (dd * dd + r * r - s * s) / (2. * dd)
        h = torch.sqrt(torch.clamp(r * r - ar * ar, min=0.))
        v = r * r * torch.atan2(h, ar) + s * s * torch.atan2(h, dd - ar) - dd * h
        area = torch.where(both, v, area)
        return torch.where(inner, torch.full_like(d, math.pi * min(r, s) ** 2), area)

    return (lens(1., 1.) - 2. * lens(1., obs) + lens(obs, obs)) / (math.pi * (1. - obs * obs))


def _kolm_k0(fwhm):
    return 2.992939911888651 / (fwhm / 0.9758634299)


def _kolm_stepk(dev):
    """stepk of the unit Kolmogorov profile (k0 = 1): GalSim's tabulated end point."""
    dlogr = (_XACC / 10.) ** 0.25
    lr = torch.arange(0, 500, dtype=torch.float64, device=dev) * dlogr - 3.
    f = _hankel(lr, torch.full_like(lr, 0.6), _contour(dev)) / torch.exp(2. * lr) / (2. * math.pi)
    r = torch.exp(lr)
    end = int(torch.nonzero(f * r * r / 1.67 < 1e-5 / (2. * math.pi))[0])
    m = 11. / 3.
    R = (2. * math.pi * float(f[end]) * float(r[end]) ** m / ((m - 2.) * _FOLD)) ** (1. / (m - 2.))
    return math.pi / max(R, _MIN_HLR * 2.992939911888651 * 0.5548101137)


def _sersic_stepk(n):
    a = 2. * n
    lo, hi = torch.zeros_like(n), torch.full_like(n, 200.)
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        up = torch.special.gammaincc(a, mid) > _FOLD
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    return math.pi / torch.clamp((0.5 * (lo + hi)) ** n, min=_MIN_HLR)


def _sersic_maxk(n, con):
    """The end of |F| > maxk_threshold on GalSim's table of ln k (units of 1 / r0)."""
    lo, hi = torch.full_like(n, -30.), torch.full_like(n, 6.3)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        up = _sersic_ft(torch.exp(2. * mid), n, con) > _MAXK
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    d6 = torch.exp(torch.special.gammaln(8. * n) - torch.special.gammaln(2. * n)) / 2304.
    front, step = torch.log(_KACC / d6) / 6. - 0.001, (_KACC / 10.) ** 0.25
    return torch.exp(front + (torch.floor((0.5 * (lo + hi) - front) / step) + 1.) * step)


def _moffat_rd(fwhm, beta):
    return fwhm / (2. * torch.sqrt(2. ** (1. / beta) - 1.))


def _moffat_sizes(beta, rd):
    e = 1. / (1. - beta)
    R = torch.minimum(_FOLD ** (0.5 * e), torch.sqrt(_XACC ** e - 1.))
    R = torch.maximum(R, _MIN_HLR * torch.sqrt(0.5 ** e - 1.)) * rd
    lo, hi = torch.zeros_like(beta), torch.full_like(beta, 60.)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        up = _moffat_ft(mid, beta) > _MAXK
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    return math.pi / R, 0.5 * (lo + hi) / rd


def _exp_stepk(r0):
    R = -math.log(_FOLD)
    for _ in range(3):
        R = math.log(1. + R) - math.log(_FOLD)
    return math.pi / max(R, _MIN_HLR * 1.6783469900166605) / r0


def _major(g1, g2):
    a = torch.sqrt(g1 * g1 + g2 * g2)
    return torch.sqrt((1. + a) / (1. - a))


def _image_sizes(stepk, maxk, nx, ny, scale, min_fft=128):
    """GalSim's (nx, ny, N, Nk) per stamp; stepk, maxk of the world profile (with its PSF)."""
    B = stepk.shape[0]
    even_x, even_y = not nx or nx % 2 == 0, not ny or ny % 2 == 0
    dr = math.hypot(0.5 if even_x else 0., 0.5 if even_y else 0.)
    stepk = math.pi / (math.pi / (stepk * scale) + dr)
    stepk = (stepk ** -2 + math.pi ** -2) ** -0.5
    maxk = np.minimum((maxk * scale).cpu().numpy(), 2000.)
    good = 2 * ((np.ceil(2. * math.pi / stepk.cpu().numpy() * (1. - 1e-12)).astype(np.int64) + 1) // 2)
    nxs = np.full(B, nx) if nx else good
    nys = np.full(B, ny) if ny else good
    need = np.maximum(np.maximum(good, 2 * (nxs // 2)), np.maximum(2 * (nys // 2), np.maximum(nxs, nys)))
    sizes = np.array(sorted([2 ** i for i in range(1, 18)] + [3 * 2 ** i for i in range(1, 17)]))
    N = np.maximum(sizes[np.searchsorted(sizes, need * (1. - 1e-5))], min_fft)
    Nk = np.where(math.pi > maxk, N, 2 * np.ceil(maxk * N / (2. * math.pi)).astype(np.int64))
    return nxs, nys, N, Nk


def _draw_exact(ft, nx, ny, N, Nk, dev, idx):
    """Stamps idx, which share (nx, ny, N, Nk): the (b, ny, nx) float64 images.  ft(idx, kx, ky) is the
    transform (complex, with phases) on pixel wave vectors."""
    hk = Nk // 2
    dk = 2. * math.pi / N
    A = torch.zeros(len(idx), N, N, dtype=torch.complex128, device=dev)
    cols = max(1, min(hk + 1, int(2.5e5 / len(idx) / (Nk + 1))))
    ky = torch.arange(-hk, hk + 1, device=dev)
    for c0 in range(0, hk + 1, cols):
        kx = torch.arange(c0, min(hk + 1, c0 + cols), device=dev)
        F = ft(idx, (kx * dk).double()[None, :, None], (ky * dk).double()[None, None, :])
        F = F * torch.where(kx == 0, 1., 2.)[None, :, None]
        at = (torch.remainder(kx, N)[:, None] * N + torch.remainder(ky, N)[None, :]).reshape(-1)
        A = A.view(len(idx), -1).index_add(1, at, F.reshape(len(idx), -1)).view(len(idx), N, N)
    img = torch.fft.ifft2(A).real                 # [x, y]
    xs = torch.remainder(torch.arange(nx, device=dev) - nx // 2, N)
    ys = torch.remainder(torch.arange(ny, device=dev) - ny // 2, N)
    return img[:, xs][:, :, ys].transpose(1, 2)


def _groups(nxs, nys, N, Nk, points=2 ** 18):
    keys = {}
    for i, k in enumerate(zip(nxs.tolist(), nys.tolist(), N.tolist(), Nk.tolist())):
        keys.setdefault(k, []).append(i)
    for k, ids in sorted(keys.items()):
        step = max(1, points // (k[3] * k[3] // 2))
        for i in range(0, len(ids), step):
            yield k, ids[i:i + step]


def _phase(kx, ky, cx, cy):
    return torch.polar(torch.ones_like(kx * cx + ky * cy), -(kx * cx + ky * cy))


def _sinc(x):
    return torch.sinc(x / (2. * math.pi))


def _centre(nx, ny):
    return (-0.5 if nx % 2 == 0 else 0.), (-0.5 if ny % 2 == 0 else 0.)


def _sheared(kx, ky, g1, g2, scale):
    f = 1. / torch.sqrt(1. - g1 * g1 - g2 * g2) / scale
    return ((1. + g1) * kx + g2 * ky) * f, (g2 * kx + (1. - g1) * ky) * f


def _fit_images(params, case, dev):
    """The fit model's images at (B, 7) parameters, differentiable (64 bits)."""
    con = _contour(dev)
    nx, ny, B = case["nx"], case["ny"], params.shape[0]
    q = params.detach().double()
    beta = torch.full((B,), 2.5, dtype=torch.float64, device=dev)
    rd = _moffat_rd(torch.full_like(beta, 0.8), beta)
    m_step, m_maxk = _moffat_sizes(beta[:1], rd[:1])
    r0 = q[:, 1] / _sersic_b(q[:, 2]) ** q[:, 2]
    gal = _sersic_stepk(q[:, 2]) / r0 / _major(q[:, 3], q[:, 4])
    gal = math.pi / (math.pi / gal + torch.hypot(q[:, 5], q[:, 6]))
    stepk = (gal ** -2 + float(m_step) ** -2 + (math.pi / SCALE) ** -2) ** -0.5
    g_maxk = _sersic_maxk(q[:, 2], con) / r0 * _major(q[:, 3], q[:, 4])
    nxs, nys, N, Nk = _image_sizes(stepk, torch.minimum(m_maxk.expand(B), g_maxk), nx, ny, SCALE)
    out = torch.zeros(B, ny, nx, dtype=torch.float64, device=dev)
    b_all = _sersic_b(params[:, 2].double())
    cx0, cy0 = _centre(nx, ny)

    def ft(ids, kx, ky):
        flux, hlr, n, g1, g2, dx, dy = [params[ids, i].double()[:, None, None] for i in range(7)]
        r0 = hlr / b_all[ids][:, None, None] ** n
        kxp, kyp = _sheared(kx, ky, g1, g2, SCALE)
        v = flux * _sersic_ft((kxp * kxp + kyp * kyp) * r0 * r0, n, con)
        k = torch.sqrt(kx * kx + ky * ky) / SCALE * rd[0]
        v = v * torch.exp(-k) * (1. + k) * (_sinc(kx) * _sinc(ky)) ** 2
        return v * _phase(kx, ky, dx / SCALE + cx0, dy / SCALE + cy0)

    if params.requires_grad:
        return ft, list(_groups(nxs, nys, N, Nk, 2 ** 17))
    for (x, y, n_, nk), ids in _groups(nxs, nys, N, Nk):
        out[ids] = _draw_exact(ft, x, y, n_, nk, dev, ids)
    return out


def _flat(case, ft, sizes, dev, B):
    """All stamps of a batch packed as draw_batch packs them, with its integer results."""
    nxs, nys, N, Nk = sizes
    off = np.concatenate([[0], np.cumsum(nxs * nys)])
    out = torch.zeros(int(off[-1]), dtype=torch.float64, device=dev)
    for (x, y, n_, nk), ids in _groups(nxs, nys, N, Nk):
        img = _draw_exact(ft, x, y, n_, nk, dev, ids)
        for j, i in enumerate(ids):
            out[off[i]:off[i + 1]] = img[j].reshape(-1)
    res = dict(pixels=out, nx=None, ny=None)
    if case.get("precision") == "fp64":
        res["added_flux"] = torch.stack([out[off[i]:off[i + 1]].sum() for i in range(B)])
    return res


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def exact(case, seed):
    kind = case["kind"]
    if kind in ("image_psf", "ccd_noise", "chromatic"):
        # an interpolated image and a random stream are defined by GalSim's own procedures
        return None
    dev = _device()
    p = _params(case, seed)
    B = p.B

    def col(a):
        return torch.as_tensor(np.atleast_1d(np.asarray(a, np.float64)), device=dev)

    nx, ny = int(case.get("nx", 0)), int(case.get("ny", 0))
    con = _contour(dev)
    if kind == "single":
        flux, hlr, fwhm = col(p.flux), col(p.hlr), col(p.fwhm)
        g1, g2 = col(p.g[0]), col(p.g[1])
        r0, beta = hlr / 1.6783469900166605, torch.full_like(hlr, 3.)
        rd = _moffat_rd(fwhm, beta)
        ms, mk = _moffat_sizes(beta, rd)
        gal = _exp_stepk(1.) / r0 / _major(g1, g2)
        gal = math.pi / (math.pi / gal + math.hypot(*p.shift))
        stepk = (gal ** -2 + ms ** -2 + (math.pi / SCALE) ** -2) ** -0.5
        sizes = _image_sizes(stepk, torch.minimum(mk, 10. / r0 * _major(g1, g2)), nx, ny, SCALE)
        cx, cy = _centre(nx, ny)

        def ft(ids, kx, ky):
            kxp, kyp = _sheared(kx, ky, g1, g2, SCALE)
            v = flux * (1. + (kxp * kxp + kyp * kyp) * r0 * r0) ** -1.5
            v = v * _moffat_ft(torch.sqrt(kx * kx + ky * ky) / SCALE * rd, beta) * (_sinc(kx) * _sinc(ky)) ** 2
            return v * _phase(kx, ky, p.shift[0] / SCALE + cx, p.shift[1] / SCALE + cy)

        (x, y, n_, nk), ids = next(_groups(*sizes))
        return dict(pixels=_draw_exact(ft, x, y, n_, nk, dev, ids)[0])
    if kind == "catalog":
        n, hlr, flux, fwhm, g1, g2 = col(p.n), col(p.hlr), col(p.flux), col(p.fwhm), col(p.g[:, 0]), col(p.g[:, 1])
        r0 = hlr / _sersic_b(n) ** n
        k0 = _kolm_k0(fwhm)
        gal = _sersic_stepk(n) / r0 / _major(g1, g2)
        stepk = (gal ** -2 + (_kolm_stepk(dev) * k0) ** -2 + (math.pi / SCALE) ** -2) ** -0.5
        maxk = torch.minimum((-math.log(_KACC)) ** 0.6 * k0, _sersic_maxk(n, con) / r0 * _major(g1, g2))
        sizes = _image_sizes(stepk, maxk, nx, ny, SCALE)
        cx, cy = _centre(nx, ny)

        def ft(ids, kx, ky):
            at = [a[ids][:, None, None] for a in (n, r0, flux, k0, g1, g2)]
            kxp, kyp = _sheared(kx, ky, at[4], at[5], SCALE)
            v = at[2] * _sersic_ft((kxp * kxp + kyp * kyp) * at[1] ** 2, at[0], con)
            v = v * torch.exp(-((kx * kx + ky * ky) / (SCALE * at[3]) ** 2) ** (5. / 6.)) * (_sinc(kx) * _sinc(ky)) ** 2
            return v * _phase(kx, ky, cx, cy)

        return _flat(case, ft, sizes, dev, B)
    if kind == "large":
        n, hlr, flux = col(p.n), col(p.hlr), col(p.flux)
        r0 = hlr / _sersic_b(n) ** n
        lod, obs = 0.1, 0.3
        a_step = math.pi / max(1. / (_FOLD * 0.5 * math.pi ** 2 * (1. - obs)), _MIN_HLR * 0.5348321477) / lod
        stepk = ((_sersic_stepk(n) / r0) ** -2 + a_step ** -2 + (math.pi / LARGE_SCALE) ** -2) ** -0.5
        # the disc's transform ends at the pixel grid's Nyquist frequency
        sizes = _image_sizes(stepk, torch.full_like(n, 0.999 * math.pi / LARGE_SCALE), 0, 0, LARGE_SCALE)

        def ft(ids, kx, ky):
            at = [a[ids][:, None, None] for a in (n, r0, flux)]
            ksq = (kx * kx + ky * ky) / LARGE_SCALE ** 2
            v = at[2] * _sersic_ft(ksq * at[1] ** 2, at[0], con)
            v = v * _airy_ft(torch.sqrt(ksq), lod, obs) * (_sinc(kx) * _sinc(ky)) ** 2
            return v * _phase(kx, ky, -0.5, -0.5)

        return _flat(case, ft, sizes, dev, B)
    if kind == "fit":
        target, isig = _target(case, p, dev)
        q = torch.as_tensor(p.pert, device=dev).double()
        img, grad = torch.zeros(B, ny, nx, dtype=torch.float64, device=dev), torch.zeros_like(q)
        ft, groups = _fit_images(q.clone().requires_grad_(True), case, dev)
        for (x, y, n_, nk), ids in groups:
            part = q[ids].clone().requires_grad_(True)
            f, _ = _fit_images(part, case, dev)
            im = _draw_exact(f, x, y, n_, nk, dev, list(range(len(ids))))
            (((im - target[ids].double()) * isig[ids].double()) ** 2).sum().backward()
            img[ids], grad[ids] = im.detach(), part.grad
        return dict(image=img, grad=grad)
    # bulge + disk: the records (float32 where they are differentiated) of the two components
    gradient = kind == "bulge_disk_grad"
    g = [col(a) for a in (p.g_b[:, 0], p.g_b[:, 1], p.g_d[:, 0], p.g_d[:, 1])]
    bh, dr0 = col(p.bh), col(p.dh) / 1.6783469900166605
    fb, fd = col(p.flux * p.bf), col(p.flux * (1. - p.bf))
    beta, four = col(p.beta), torch.full((B,), 4., dtype=torch.float64, device=dev)
    rd = _moffat_rd(col(p.fwhm), beta)
    ms, mk = _moffat_sizes(beta, rd)
    r0 = bh / _sersic_b(four) ** four
    step = torch.minimum(_sersic_stepk(four) / r0 / _major(g[0], g[1]), _exp_stepk(1.) / dr0 / _major(g[2], g[3]))
    stepk = (step ** -2 + ms ** -2 + (math.pi / SCALE) ** -2) ** -0.5
    # (the bulge's maxk is far above the PSF's)
    sizes = _image_sizes(stepk, mk, nx, ny, SCALE, 32)
    cx, cy = _centre(nx, ny) if nx else (-0.5, -0.5)

    def jac(g1, g2):
        f = 1. / torch.sqrt(1. - g1 * g1 - g2 * g2) / SCALE
        return torch.stack([(1. + g1) * f, g2 * f, g2 * f, (1. - g1) * f], -1)

    rec = [fb, jac(g[0], g[1]), bh, four, fd, jac(g[2], g[3]), dr0]
    if gradient:
        rec = [r.float().double() for r in rec]
    mix = [rd, beta]
    if gradient:
        mix = [rd.float().double(), beta]

    def make_ft(rec):
        r_e = _sersic_b(rec[3]) ** rec[3]

        def ft(ids, kx, ky):
            fb, jb, hb, nb, fd, jd, rdisk = [r[ids] for r in rec]
            kk = []
            for j in (jb, jd):
                j = j[:, :, None, None]
                kk.append((j[:, 0] * kx + j[:, 2] * ky) ** 2 + (j[:, 1] * kx + j[:, 3] * ky) ** 2)
            fb, hb, nb, fd, rdisk, re = [a[:, None, None] for a in (fb, hb, nb, fd, rdisk, r_e[ids])]
            v = fb * _sersic_ft(kk[0] * (hb / re) ** 2, nb, con) + fd * (1. + kk[1] * rdisk * rdisk) ** -1.5
            m = _moffat_ft(torch.sqrt(kx * kx + ky * ky) / SCALE * mix[0][ids_of[0]][ids][:, None, None],
                           mix[1][ids_of[0]][ids][:, None, None])
            return v * m * (_sinc(kx) * _sinc(ky)) ** 2 * _phase(kx, ky, cx, cy)

        return ft

    ids_of = [list(range(B))]
    if not gradient:
        return _flat(case, make_ft(rec), sizes, dev, B)
    L = 5
    out = dict(image=torch.zeros(B, ny, nx, dtype=torch.float64, device=dev),
               leaf_flux=torch.zeros(B, L, dtype=torch.float64, device=dev),
               leaf_jac=torch.zeros(B, L, 4, dtype=torch.float64, device=dev),
               leaf_size=torch.zeros(B, L, 2, dtype=torch.float64, device=dev),
               leaf_n=torch.zeros(B, L, dtype=torch.float64, device=dev))
    cot = torch.as_tensor(p.cot, device=dev).double()
    for (x, y, n_, nk), ids in _groups(*sizes, points=2 ** 17):
        ids_of[0] = ids
        part = [r[ids].clone().requires_grad_(True) for r in rec]
        im = _draw_exact(make_ft(part), x, y, n_, nk, dev, list(range(len(ids))))
        (im * cot[ids]).sum().backward()
        out["image"][ids] = im.detach()
        d = [r.grad for r in part]
        out["leaf_flux"][ids, 0], out["leaf_flux"][ids, 1] = d[0], d[4]
        out["leaf_jac"][ids, 0], out["leaf_jac"][ids, 1] = d[1], d[5]
        out["leaf_size"][ids, 0, 0], out["leaf_size"][ids, 1, 0] = d[2], d[6]
        out["leaf_n"][ids, 0] = d[3]
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------
#: Typical FFT size, stamp side (automatic) and arithmetic per wave vector of each kind.
_TYPICAL = dict(single=(128, 0, 40), catalog=(140, 105, 60), image_psf=(136, 0, 150), fit=(128, 0, 200),
                bulge_disk=(96, 62, 120), bulge_disk_grad=(96, 0, 250), large=(7000, 5500, 80),
                chromatic=(128, 0, 300), ccd_noise=(0, 0, 0))


def work(case):
    N, auto, per_k = _TYPICAL[case["kind"]]
    B = int(case.get("stamps", 1))
    pixels = B * (case["nx"] * case["ny"] if case.get("nx") else auto * auto)
    size = 8 if case.get("precision") == "fp64" or case["kind"] == "single" else 4
    if case["kind"] == "ccd_noise":
        return dict(bytes=2. * 4. * pixels, flops=60. * pixels)
    ffts = 2 if case["kind"] in ("fit", "bulge_disk_grad", "chromatic") else 1
    flops = B * (per_k * N * N / 2. + ffts * 2.5 * N * N * 2. * math.log2(N))
    return dict(bytes=float(pixels * size * ffts + B * 60.), flops=float(flops))
