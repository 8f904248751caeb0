"""The draws of tests/golden/double_image_fp32.npz: float arithmetic (drawImage's default) into double images."""


def cases(galsim):
    """(name, object, nx, ny): every profile kind, several Sersic indices, a sum, and a large FFT."""
    def sheared(obj):
        return obj.shear(g1=0.12, g2=-0.07).shift(0.11, -0.06)

    pix = galsim.Pixel(0.2)
    moffat = galsim.Moffat(beta=3.2, fwhm=0.7)
    for n in (0.7, 1.6, 2.5, 4.):
        gal = sheared(galsim.Sersic(n=n, half_light_radius=0.8, flux=3.))
        yield 'sersic_%.1f' % n, galsim.Convolve(gal, galsim.Kolmogorov(fwhm=0.7), pix), 25, 18
    yield 'sersic_moffat', galsim.Convolve(sheared(galsim.Sersic(n=2., half_light_radius=0.5)), moffat), 24, 21
    yield 'exponential', galsim.Convolve(sheared(galsim.Exponential(half_light_radius=0.8)), moffat, pix), 24, 20
    yield 'moffat', sheared(galsim.Moffat(beta=2.5, fwhm=0.9)), 20, 20
    yield 'airy', galsim.Convolve(sheared(galsim.Exponential(half_light_radius=0.5)),
                                  galsim.Airy(lam_over_diam=0.2, obscuration=0.3)), 20, 20
    yield 'sum', galsim.Convolve(galsim.Add(sheared(galsim.Sersic(n=3., half_light_radius=0.5, flux=2.)),
                                            sheared(galsim.Exponential(half_light_radius=1.))), moffat, pix), 26, 22
    gsp = galsim.GSParams(minimum_fft_size=2048)
    yield 'large', galsim.Convolve(sheared(galsim.Sersic(n=1.5, half_light_radius=0.8, gsparams=gsp)),
                                   galsim.Kolmogorov(fwhm=0.7, gsparams=gsp)), 20, 20
