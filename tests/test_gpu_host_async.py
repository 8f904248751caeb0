"""StampBatch.host_async: the read-back on a copy stream returns the same pixels as host(),
for reads in flight while the next batch is drawn (the pipelined catalog loop)."""
import numpy as np
import pytest

import galsim_b200 as galsim

pytestmark = pytest.mark.gpu


def _obj(seed):
    rng = np.random.default_rng(seed)
    n = 16
    gal = galsim.Sersic(n=rng.uniform(0.8, 3.5, n), half_light_radius=rng.uniform(0.3, 1.0, n),
                        flux=1e3).shear(g1=rng.uniform(-0.2, 0.2, n), g2=0.05)
    return galsim.Convolve(gal, galsim.Kolmogorov(fwhm=0.7), galsim.Pixel(0.2))


def test_pipelined_reads_match_synchronous_reads():
    pending, expected, fluxes = [], [], []
    for seed in range(4):
        sb = galsim.draw_batch(_obj(seed), scale=0.2, dtype=np.float32)
        expected.append(sb.host(copy=True))
        fluxes.append(sb.added_flux)
        pending.append(sb.host_async())
        if len(pending) == 2:
            r = pending.pop(0)
            np.testing.assert_array_equal(r.result(), expected[seed - 1])
            np.testing.assert_array_equal(r.added_flux(), fluxes[seed - 1])
    r = pending.pop(0)
    np.testing.assert_array_equal(r.result(), expected[-1])
    np.testing.assert_array_equal(r.added_flux(), fluxes[-1])


@pytest.mark.parametrize('fixed', [False, True])
def test_draw_batches_matches_draw_batch(fixed):
    """draw_batches (next batch planned on a worker thread, reads on a copy stream) yields every
    batch's pixels and fluxes exactly as draw_batch draws them, in order."""
    size = dict(nx=40, ny=40) if fixed else {}
    expected = []
    for seed in range(5):
        sb = galsim.draw_batch(_obj(seed), scale=0.2, dtype=np.float32, **size)
        expected.append((sb.host(copy=True), np.array(sb.added_flux), list(sb.offsets)))
    got = [(sb, pix.copy(), flux.copy()) for sb, pix, flux in
           galsim.draw_batches((_obj(seed) for seed in range(5)), scale=0.2, dtype=np.float32, **size)]
    assert len(got) == len(expected)
    for (sb, pix, flux), (epix, eflux, eoff) in zip(got, expected):
        assert list(sb.offsets) == eoff
        np.testing.assert_array_equal(pix, epix)
        np.testing.assert_array_equal(flux, eflux)


def test_draw_batches_empty_sequence():
    assert list(galsim.draw_batches(iter(()), scale=0.2)) == []


def _tableless_obj(seed):
    """Leaves without tables: nothing in the sizing waits for a table build."""
    rng = np.random.default_rng(seed)
    n = 300
    gal = galsim.Exponential(half_light_radius=rng.uniform(0.3, 1.0, n), flux=rng.uniform(1., 9., n)) \
        .shear(g1=rng.uniform(-0.2, 0.2, n), g2=0.05)
    return galsim.Convolve(gal, galsim.Moffat(beta=rng.uniform(2., 4., n), fwhm=0.7), galsim.Pixel(0.2))


def test_draw_batches_on_a_stream_of_the_callers():
    """The worker thread plans on its own current stream, the batches run on the caller's."""
    import torch
    expected = [galsim.draw_batch(_tableless_obj(seed), nx=40, ny=40, scale=0.2).host(copy=True) for seed in range(4)]

    def objects():
        for seed in range(4):
            torch.cuda._sleep(20000000)      # the default stream is behind when the records are uploaded
            yield _tableless_obj(seed)

    with torch.cuda.stream(torch.cuda.Stream()):
        got = [pix.copy() for _, pix, _ in galsim.draw_batches(objects(), nx=40, ny=40, scale=0.2)]
    for a, b in zip(got, expected):
        np.testing.assert_array_equal(a, b)


def test_a_plan_made_under_another_stream():
    import torch
    expected = galsim.draw_batch(_tableless_obj(7), nx=40, ny=40, scale=0.2).host(copy=True)
    planned, run = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(planned):
        torch.cuda._sleep(50000000)
        plan = galsim.plan_batch(_tableless_obj(7), nx=40, ny=40, scale=0.2)
    with torch.cuda.stream(run):
        sb = galsim.run_batch(plan)
        del plan                             # its memory is not handed out again while `run` reads it
        with torch.cuda.stream(planned):
            junk = [torch.full((300 * 3 * 136,), 255, dtype=torch.uint8, device='cuda') for _ in range(4)]
        got = sb.host(copy=True)
    del junk
    np.testing.assert_array_equal(got, expected)
