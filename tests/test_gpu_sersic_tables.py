"""GPU: the Sersic table kernel's variants -- one node a thread (small builds) and three (large ones),
ln k grids up to the resampled levels' spacing and wider -- against the oracle's table of the same n,
and against each other through the draws and gradients that read the nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

import galsim_b200 as galsim  # noqa: E402
import galsim_oracle as O  # noqa: E402

H = dict(N=0, NUSED=1, KSQMAX=5, HIGHA=8, HIGHB=9, MAXK=10, STATUS=15)


@pytest.mark.parametrize('with_dn', [False, True])
@pytest.mark.parametrize('spacing', [1., 2.5])
@pytest.mark.parametrize('count', [3, 700])
def test_tables_against_the_oracle(count, spacing, with_dn):
    from galsim_b200 import _lib
    check = (0.3, 0.95, 2.6)
    n = np.unique(np.concatenate([check, np.linspace(0.4, 2.5, count - 3)]))
    t = _lib.Tables()
    t.build_sersic(n, galsim.GSParams(table_spacing=spacing), with_dn=with_dn)
    head = t.sersic_info()
    assert not head[:, H['STATUS']].any()
    for c in check:
        info = O.SersicInfo(c, O.OGSParams(table_spacing=spacing))
        h = head[np.flatnonzero(n == c)[0]]
        # the stop and maxk are nodes of the grid; the fit's nodes are a few 1e-5 of the flux and
        # agree to ~1e-11 of it, and the fit over a span of 0.3 in ln k amplifies that ~10 times
        np.testing.assert_allclose(h[H['KSQMAX']], info.ksq_max, rtol=1e-12)
        np.testing.assert_allclose(h[H['MAXK']], info.maxk, rtol=1e-12)
        np.testing.assert_allclose(h[H['HIGHA']], info.highk_a, rtol=1e-5)
        np.testing.assert_allclose(h[H['HIGHB']], info.highk_b, rtol=1e-4)


@pytest.mark.parametrize('spacing', [1., 2.5])
def test_large_build_draws_and_differentiates_as_small_builds(spacing):
    from galsim_b200 import autodiff
    gsp = galsim.GSParams(table_spacing=spacing)
    rng = np.random.default_rng(5)
    B = 650
    p = np.stack([rng.uniform(1., 9., B), rng.uniform(0.3, 0.8, B), rng.uniform(0.35, 5.5, B), rng.normal(0., 0.1, B),
                  rng.normal(0., 0.1, B), rng.normal(0., 0.1, B), rng.normal(0., 0.1, B)], -1)
    psf = galsim.Gaussian(sigma=0.4, gsparams=gsp)
    cot = torch.as_tensor(rng.standard_normal((B, 31, 32)), device='cuda')
    some = [0, 1, 311, 648, 649]

    def run(rows):
        model = autodiff.GalaxyModel(psf, 32, 31, 0.2, dtype=np.float64, precision='fp64', gsparams=gsp)
        q = torch.as_tensor(p[rows], device='cuda').requires_grad_(True)
        img = model(q)
        img.backward(cot[rows])
        return img.detach().cpu().numpy(), q.grad.cpu().numpy()

    img, grad = run(list(range(B)))
    simg, sgrad = run(some)
    # node sums in another order: ~1e-15 of the terms' size, up to ~1e-11 of the flux after the
    # levels' own cancellation
    np.testing.assert_allclose(img[some], simg, rtol=0, atol=1e-10 * np.abs(simg).max())
    np.testing.assert_allclose(grad[some], sgrad, rtol=0, atol=1e-8 * np.abs(sgrad).max())


def test_levels_are_resampled_as_builds_need_them():
    """A first build of a spacing spreads the quadrature levels its nodes ask for, not all 57 (which take over 40 ms;
    these about 1); a later build that needs more adds them and leaves what is there as it is."""
    import time
    from galsim_b200 import _lib

    def build(n, gsp):
        tb = _lib.Tables()
        torch.cuda.synchronize()
        t = time.perf_counter()
        tb.build_sersic(np.array([n]), gsp)
        torch.cuda.synchronize()
        return time.perf_counter() - t, tb.sersic_info()[0]

    build(2., galsim.GSParams())                             # (loads the kernels)
    first = [build(2., galsim.GSParams(table_spacing=s))[0] for s in (0.8137, 0.8138, 0.8139, 0.814)]
    assert min(first) < 0.02
    gsp = galsim.GSParams(table_spacing=0.8137)              # (evicted or not)
    info = build(2., gsp)[1]
    assert build(5., gsp)[1][H['STATUS']] == 0
    assert np.array_equal(build(2., gsp)[1], info)
    # an accuracy whose nodes ask for more levels than the rule expects gets them
    _, tight = build(2., galsim.GSParams(table_spacing=0.8137, integration_relerr=1e-10, integration_abserr=1e-13))
    assert tight[H['STATUS']] == 0 and tight[H['NUSED']] == info[H['NUSED']]


@pytest.mark.parametrize('spacing', [1., 0.3, 2.5])
def test_a_table_does_not_depend_on_the_others_of_its_build(spacing):
    """Small builds take one node a thread and large ones three: the same numbers, in the tables' constants and in
    double-precision stamps drawn from them."""
    from galsim_b200 import _lib
    gsp = galsim.GSParams(table_spacing=spacing)
    few = np.array([0.5, 1.3, 2.6, 4., 6.1])
    many = np.unique(np.concatenate([few, np.linspace(0.4, 3.9, 800)]))
    heads = []
    for n in (few, many):
        t = _lib.Tables()
        t.build_sersic(n, gsp, with_dn=True)
        heads.append(t.sersic_info()[[int(np.flatnonzero(n == v)[0]) for v in few]])
    assert np.array_equal(heads[0], heads[1])
    stamps = []
    for n in (few[:4], many[many < 4.01]):
        obj = galsim.Convolve(galsim.Sersic(n=n, half_light_radius=np.full(len(n), 0.6), gsparams=gsp), galsim.Gaussian(sigma=0.3))
        sb = galsim.draw_batch(obj, nx=24, ny=24, scale=0.2, dtype=np.float64, precision='fp64')
        a = sb.host(copy=True).reshape(len(n), 24, 24)
        stamps.append(a[[int(np.flatnonzero(n == v)[0]) for v in few[:4]]])
    assert np.array_equal(stamps[0], stamps[1])


@pytest.mark.parametrize('count', [3, 700])
@pytest.mark.parametrize('spacing', [0.3, 0.55])
def test_fine_tables_against_the_oracle(count, spacing):
    """ln k grids finer than the resampled levels' spacing: one level point in three or one in one node."""
    test_tables_against_the_oracle(count, spacing, False)
