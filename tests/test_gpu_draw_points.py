"""GPU: the draw kernels' evaluation of several wave vectors a lane (leaf kinds with constants in the
working precision, the fold over a column's aliases, the last point of columns with Nk a multiple of
32) against the FP64 path, which takes the general form, over FFT sizes, aliasing and profile types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip('torch')

import galsim_b200 as galsim  # noqa: E402


def _profiles(gsp, B):
    rng = np.random.default_rng(11)
    g1, g2 = rng.uniform(-0.2, 0.2, B), rng.uniform(-0.2, 0.2, B)
    ones = np.ones(B)
    return {
        'exponential': galsim.Exponential(scale_radius=1.2 * ones, gsparams=gsp).shear(g1=g1, g2=g2),
        'sersic': galsim.Sersic(n=rng.uniform(0.6, 4., B), half_light_radius=1.5 * ones, gsparams=gsp).shear(g1=g1, g2=g2),
        'moffat': galsim.Moffat(beta=rng.uniform(1.6, 6., B), fwhm=1.7 * ones, gsparams=gsp).shear(g1=g1, g2=g2),
        'moffat_half': galsim.Moffat(beta=np.where(np.arange(B) % 2, 2.5, 3.5), fwhm=1.7 * ones, gsparams=gsp),
        'kolmogorov': galsim.Kolmogorov(fwhm=1.7 * ones, gsparams=gsp).shear(g1=g1, g2=g2),
        'airy': galsim.Airy(lam_over_diam=1.1 * ones, obscuration=0.3, gsparams=gsp).shear(g1=g1, g2=g2),
        'gaussian': galsim.Gaussian(sigma=0.8 * ones, gsparams=gsp).shear(g1=g1, g2=g2),
    }


@pytest.mark.parametrize('min_n,scale', [(32, 1.), (48, 1.), (64, 0.6), (96, 1.7), (128, 1.3), (192, 1.), (256, 2.2),
                                         (384, 1.), (1024, 1.)])
@pytest.mark.parametrize('kind', ['exponential', 'sersic', 'moffat', 'moffat_half', 'kolmogorov', 'airy', 'gaussian',
                                  'sum'])
def test_float_draws_against_double(kind, min_n, scale):
    B = 3
    gsp = galsim.GSParams(minimum_fft_size=min_n, folding_threshold=0.05, stepk_minimum_hlr=1.)
    p = _profiles(gsp, B)
    obj = p[kind] if kind != 'sum' else galsim.Add(p['sersic'] * 0.4, p['exponential'] * 0.6)
    obj = galsim.Convolve(obj, galsim.Gaussian(sigma=0.4, gsparams=gsp)).shift(0.3, -0.2)
    lo, hi = [galsim.draw_batch(obj, nx=25, ny=18, scale=scale, dtype=np.float64 if q == 'fp64' else np.float32, precision=q)
              for q in ('fp32', 'fp64')]
    assert np.array_equal(lo.N, hi.N) and np.array_equal(lo.Nk, hi.Nk)
    a, b = lo.flat.cpu().numpy().reshape(B, 18, 25).astype(float), hi.flat.cpu().numpy().reshape(B, 18, 25)
    # single precision: a few 1e-7 of the value a wave vector, summed over the image with random signs
    for x, y in zip(a, b):
        assert np.abs(x - y).max() <= 3e-6 * np.abs(y).max()


def test_double_image_keeps_the_general_path():
    """drawImage into a double image at the default precision: one object and a batch agree bit for bit."""
    obj = galsim.Convolve(galsim.Exponential(flux=3., half_light_radius=0.8).shear(g1=0.1, g2=-0.05),
                          galsim.Moffat(beta=3., fwhm=0.7), galsim.Pixel(0.2))
    im = obj.drawImage(galsim.ImageD(48, 40), scale=0.2, method='fft')
    many = galsim.Convolve(galsim.Exponential(flux=np.full(3, 3.), half_light_radius=0.8).shear(g1=0.1, g2=-0.05),
                           galsim.Moffat(beta=3., fwhm=0.7), galsim.Pixel(0.2))
    sb = galsim.draw_batch(many, nx=48, ny=40, scale=0.2, dtype=np.float64, precision='fp32')
    for a in sb.flat.cpu().numpy().reshape(3, 40, 48):
        assert np.array_equal(a, im.array)


@pytest.mark.parametrize('n', [192, 256, 384, 768, 1024, 1536, 2048, 4096, 6144, 8192, 12288])
def test_one_object_into_a_double_image_by_the_split_path(n):
    gsp = galsim.GSParams(minimum_fft_size=n, maximum_fft_size=16384, folding_threshold=0.05, stepk_minimum_hlr=1.)
    obj = galsim.Convolve(galsim.Exponential(flux=np.full(1, 3.), half_light_radius=0.8, gsparams=gsp).shear(g1=0.1, g2=-0.05),
                          galsim.Moffat(beta=3., fwhm=0.7, gsparams=gsp), galsim.Pixel(0.2, gsparams=gsp))
    lo, hi = [galsim.draw_batch(obj, nx=41, ny=30, scale=0.2, dtype=np.float64, precision=q) for q in ('fp32', 'fp64')]
    assert lo.N[0] == n == hi.N[0]
    a, b = lo.flat.cpu().numpy(), hi.flat.cpu().numpy()
    # single precision: a few 1e-7 of the value a wave vector, summed over the image with random signs
    assert np.abs(a - b).max() <= 3e-6 * np.abs(b).max()


MODES = {'float': ('fp32', np.float32), 'float into double': ('fp32', np.float64), 'double': ('fp64', np.float64)}


# (FFT size, pixel scale): Nk = N at 0.2, several times N at the larger scales
@pytest.mark.parametrize('min_n,scale', [(192, 0.2), (192, 1.), (256, 2.2), (384, 1.), (512, 0.2), (768, 1.5), (1024, 0.2),
                                         (1024, 1.)])
@pytest.mark.parametrize('mode', sorted(MODES))
def test_fused_and_split_kernels_give_the_same_bits(mode, min_n, scale):
    """Which of the two a bucket runs on is chosen by a timing, so it must not show in the pixels."""
    from galsim_b200 import _lib
    B = 3
    gsp = galsim.GSParams(minimum_fft_size=min_n, folding_threshold=0.05, stepk_minimum_hlr=1., maximum_fft_size=1 << 15)
    p = _profiles(gsp, B)
    y, x = np.mgrid[:24, :24] - 11.5
    psf = galsim.InterpolatedImage(galsim.Image((1. + (x * x + 1.1 * y * y) / 4.) ** -3., scale=0.35), gsparams=gsp)
    p['sum'] = galsim.Convolve(galsim.Add(p['sersic'] * 0.4, p['exponential'] * 0.6), p['moffat'])
    p['image'] = galsim.Convolve(p['sersic'], psf)
    p['tree'] = galsim.Add(galsim.Convolve(p['exponential'], p['kolmogorov']), p['moffat'].shift(0.2, 0.1))
    precision, dtype = MODES[mode]
    for kind, obj in p.items():
        obj = galsim.Convolve(obj, galsim.Gaussian(sigma=0.4, gsparams=gsp)).shift(0.3, -0.2)
        got = []
        try:
            for variant in (1, 2):
                _lib.set_draw_variant(variant)
                got.append(galsim.draw_batch(obj, nx=25, ny=18, scale=scale, dtype=dtype, precision=precision))
        finally:
            _lib.set_draw_variant(0)
        assert got[0].N.min() >= min_n
        assert np.array_equal(got[0].host(copy=True), got[1].host(copy=True)), kind


@pytest.mark.parametrize('mode', sorted(MODES))
def test_a_first_draw_equals_the_next_ones(mode):
    """The call that times the two kernels returns what later calls return."""
    precision, dtype = MODES[mode]
    hlr = np.linspace(1., 2.5, 37)
    obj = galsim.Convolve(galsim.Exponential(half_light_radius=hlr).shear(g1=0.1, g2=0.2), galsim.Kolmogorov(fwhm=0.7))
    a = [galsim.draw_batch(obj, nx=150, ny=130, scale=0.2, dtype=dtype, precision=precision) for _ in range(3)]
    assert a[0].N.min() >= 192        # (two kernels to choose from)
    for b in a[1:]:
        assert np.array_equal(a[0].host(copy=True), b.host(copy=True))


def test_double_images_are_those_of_the_general_forms():
    """Float arithmetic into a double image: every profile takes its general form, so the pixels are those
    stored in double_image_fp32.npz, drawn by the tree of commit b079620, which knew no other.  A Sersic table
    is within 1e-12 of that tree's, which can turn the rounding of one of its ~250 FP32 nodes, 6e-8 of its
    share: 1e-8 of the peak."""
    import os
    from double_image_cases import cases
    gold = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), 'golden', 'double_image_fp32.npz'))
    for name, obj, nx, ny in cases(galsim):
        a = obj.drawImage(galsim.ImageD(nx, ny), scale=0.2, method='fft').array
        assert np.abs(a - gold[name]).max() <= 1e-8 * gold[name].max(), name


@pytest.mark.parametrize('kind', ['exponential', 'sersic', 'moffat', 'moffat_half', 'kolmogorov', 'sersic_kolmogorov'])
def test_float_forms_are_as_exact_as_the_general_ones(kind):
    """rms error of float images against double: the fast forms' against that of the general forms (which a
    double image takes; rounded to float here), over FFT sizes and pixel scales.  Not larger, with a tenth for
    the scatter of the ratio (13 sizes of three images, whose roundings the two share in part)."""
    ratio = []
    for min_n, scale in [(64, 1.), (64, 0.2), (96, 0.7), (128, 1.3), (128, 0.2), (192, 1.), (192, 0.2), (256, 0.6), (384, 1.),
                         (512, 0.2), (768, 0.4), (1024, 0.2), (2048, 0.2)]:
        gsp = galsim.GSParams(minimum_fft_size=min_n, folding_threshold=0.05, stepk_minimum_hlr=1., maximum_fft_size=1 << 15)
        p = _profiles(gsp, 3)
        p['sersic_kolmogorov'] = galsim.Convolve(p['sersic'], galsim.Kolmogorov(fwhm=0.7, gsparams=gsp))
        obj = galsim.Convolve(p[kind], galsim.Gaussian(sigma=0.4, gsparams=gsp)).shift(0.3, -0.2)
        fast, general, exact = [galsim.draw_batch(obj, nx=41, ny=30, scale=scale, dtype=d, precision=q).host(copy=True)
                                for q, d in (('fp32', np.float32), ('fp32', np.float64), ('fp64', np.float64))]
        ratio.append(np.sqrt(np.mean((fast - exact) ** 2) / np.mean((general.astype(np.float32) - exact) ** 2)))
    assert np.exp(np.mean(np.log(ratio))) <= 1.1, ratio


@pytest.mark.parametrize('kind', ['kolmogorov', 'sersic', 'exponential'])
def test_wave_vectors_whose_square_overflows(kind):
    """A profile so large that k^2 in its units is beyond float's range: its value there is 0, as in double."""
    from galsim_b200 import _lib
    big = np.full(2, 1e22)
    obj = {'kolmogorov': lambda: galsim.Kolmogorov(fwhm=big), 'sersic': lambda: galsim.Sersic(n=1.5, half_light_radius=big),
           'exponential': lambda: galsim.Exponential(half_light_radius=big)}[kind]()
    img = []
    for precision, dt in ((_lib.F32, _lib.F32), (_lib.F64, _lib.F64)):
        prog = galsim.plan_batch(obj, nx=20, ny=20, scale=0.2).prog
        n = np.full(2, 64)
        img.append(prog.draw_stamps(n, n, -10, -10, 20, 20, dt, precision=precision)[0].double().cpu().numpy())
    assert np.all(np.isfinite(img[0])) and img[1].max() > 0.
    assert np.abs(img[0] - img[1]).max() <= 1e-6 * img[1].max()
