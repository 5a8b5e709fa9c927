"""The clipper in blocks of spectra (csrc/rfi_blocks.cuh) against the oracle's
FP64 variant, bit for bit: data, flags and state.

The cases are those where a block cannot be done in one go: blocks' ends
(2048 spectra) inside a call and calls of a few spectra; the histories filling
inside a block; averages that sit at a binade's end (a level of 8192) or are
0, infinite or NaN; narrowband channels whose values reach down to the margin
while the averages drift, so that expected and exact margins clip different
channels; channels that get their last good value late; a bandpass with terms
and killed channels, binned from another channel count; spectra rejected for
good, up to the statistics' reset.
"""
import numpy as np
import pytest

from gen import make_bp_text, stokes_filterbank

pytestmark = pytest.mark.gpu

START, WIDTH = 140.0, 0.01220703125


def _run(pv, oracle, cuda, data, cuts, bp, history, zero_dm=True, cr=5.0, sr=4.0):
    import torch
    nbins = data.shape[1] * data.shape[3]
    kw = dict(cr=cr, sr=sr, history=history, zero_dming=zero_dm)
    g = pv.RFI(bp, **kw)
    o = oracle.RFI(bp, mode=1, parts=pv.load().pv_rfi_parts(nbins), **kw)
    a = 0
    for b in list(cuts) + [data.shape[0]]:
        d = np.ascontiguousarray(data[a:b])
        dd = torch.from_numpy(d).to(cuda)
        gf = g.run(dd, flags=True).cpu().numpy()
        of = o.run(d, flags=True)
        assert np.array_equal(gf, of), (a, b, np.argwhere(gf != of)[:4])
        assert np.array_equal(dd.cpu().numpy(), d, equal_nan=True), (a, b)
        a = b
    gs, os_ = g.state(), o.state()
    k = [0, 1, 5, 6, 7, 8, 9]
    assert np.array_equal(gs[k], os_[k], equal_nan=True)


@pytest.mark.parametrize("nsub,nchan,history,cuts", [
    (4, 16, 1000, (1, 3, 2051)),        # 64 channels, 256 partials; calls of 1 and 2 spectra
    (65, 16, 1500, (2048,)),            # 1040: 512 partials
    (8, 16, 4000, ()),                  # the histories fill in the second block
    (8, 16, 5, (700,)),                 # a history shorter than a group: every spectrum clipped
])
def test_blocks_and_calls(pv, oracle, cuda, nsub, nchan, history, cuts):
    rng = np.random.default_rng(nsub + history)
    data = stokes_filterbank(rng, 4500, nsub, nchan)
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, cuts, bp, history)


@pytest.mark.parametrize("nbins,channels", [(8200, 8), (16392, 8)])
def test_wide_bands(pv, oracle, cuda, nbins, channels):
    """9 to 16 channels per thread, and more (read again instead of kept)."""
    rng = np.random.default_rng(nbins)
    data = stokes_filterbank(rng, 1200, nbins // channels, channels)
    bp = make_bp_text(nbins, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, (1100,), bp, 1050)


@pytest.mark.parametrize("level,drift", [(8192.0, 0.0), (8192.0, 2e-4), (1000.0, -2e-4)])
def test_margin_inside_the_narrowband_values(pv, oracle, cuda, level, drift):
    """Channels whose values scatter around the margin (some proofs fail, or
    most of a block's), a mean at a binade's end, drifting levels."""
    rng = np.random.default_rng(int(level) + int(1e6 * abs(drift)))
    nt, nsub, nchan = 6000, 16, 16
    x = np.abs(rng.normal(level, level / 4, (nt, nsub * nchan))) + 64.0
    x[:, rng.choice(nsub * nchan, 12, replace=False)] *= rng.uniform(2.0, 30.0, 12)
    x *= np.exp(drift * np.arange(nt))[:, None]
    x[rng.integers(0, nt, 3)] *= 3.0
    data = x.astype(np.float32).reshape(nt, nsub, 1, nchan)
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, (1500,), bp, 1200)


def test_last_good_values_filled_late(pv, oracle, cuda):
    """Channels that are clipped for the first thousands of spectra and fill
    one by one inside a block, others that stay 0."""
    rng = np.random.default_rng(5)
    nt, nsub, nchan = 4300, 8, 16
    data = stokes_filterbank(rng, nt, nsub, nchan, rfi_channels=0.0).reshape(nt, -1)
    for n, c in enumerate(rng.choice(nsub * nchan, 9, replace=False)):
        data[:1300 + 170 * n, c] *= 40.0
        data[1300 + 170 * n + 40::7, c] *= 40.0
    data[:, 17] = 0.0
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data.reshape(nt, nsub, 1, nchan), (1100,), bp, 1050)


@pytest.mark.parametrize("nbins_file,kill", [(256, False), (1024, False), (512, True)])
def test_bandpass_with_terms(pv, oracle, cuda, nbins_file, kill):
    """A polynomial bandpass rebinned by 2 and 1/2 (half-way sums of its
    level), and one with a killed channel."""
    rng = np.random.default_rng(nbins_file)
    nt, nsub, nchan = 3000, 32, 16
    f = START + WIDTH * np.arange(512)
    data = stokes_filterbank(rng, nt, nsub, nchan, shape=1000.0 + 0.3 * f - 0.0011 * f * f)
    bp = make_bp_text(nbins_file, START, WIDTH * 512 / nbins_file, 1000.0, 50.0, (0.3, -0.0011))
    if kill:  # a kill line names a bin whose index is also its frequency
        n = int(round((149.0 - START) / WIDTH))
        bp = make_bp_text(512, 0.0, 1.0, 1000.0, 50.0, (0.3, -0.0011)) + "K 7 7\n"
        assert n > 0
    _run(pv, oracle, cuda, data, (1400,), bp, 1200)


def test_values_that_are_not_finite(pv, oracle, cuda):
    rng = np.random.default_rng(11)
    nt, nsub, nchan = 2600, 4, 16
    data = stokes_filterbank(rng, nt, nsub, nchan)
    data[1700, 1, 0, 3] = np.inf
    data[1900, 2, 0, 5] = np.nan
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, (), bp, 1100)


def test_zero_data(pv, oracle, cuda):
    data = np.zeros((2300, 4, 1, 16), np.float32)
    bp = make_bp_text(64, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, (), bp, 1100)


def test_rejected_until_the_reset(pv, oracle, cuda):
    """Every spectrum after the first 1000 rejected: the statistics of the
    second ten histories reset the averages."""
    rng = np.random.default_rng(13)
    nt, nsub, nchan = 21500, 4, 16
    data = stokes_filterbank(rng, nt, nsub, nchan, rfi_channels=0.0, burst_rate=0.0)
    data[1005:] *= 3.0
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, (9000,), bp, 1000, sr=0.5)


@pytest.mark.parametrize("hits,history", [(2, 2500), (30, 2500), (3000, 2500), (30, 1100)])
def test_few_and_many_failures_with_full_histories(pv, oracle, cuda, hits, history):
    """Spectra with a fifth of their channels scattered around the margin: a
    block with one or two failed proofs goes on by itself, one with many is
    forecast from the first of them on, in one go or (a history shorter than
    the block) in several."""
    rng = np.random.default_rng(hits + history)
    nt, nsub, nchan = history + 4200, 8, 16
    x = rng.normal(1000.0, 30.0, (nt, nsub * nchan))
    for t in history + 10 + rng.choice(nt - history - 10, hits, replace=False):
        c = rng.choice(nsub * nchan, nsub * nchan // 5, replace=False)
        x[t, c] += rng.uniform(0.0, 2500.0, c.size)
    x *= np.linspace(1.0, 1.05, nt)[:, None]
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, x.astype(np.float32).reshape(nt, nsub, 1, nchan), (history,), bp, history)


@pytest.mark.parametrize("nsub,few", [(8, 4), (65, 4), (320, 2)])
def test_few_spectra_take_one_launch(pv, oracle, cuda, nsub, few):
    """Calls of a few spectra, and the few left of a call after its last whole
    block, are walked: one launch, bit for bit the same."""
    import torch
    nt, nchan = 2 * 2048 + few + 1, 16
    data = stokes_filterbank(np.random.default_rng(nsub), nt, nsub, nchan)
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    _run(pv, oracle, cuda, data, (1, 1 + few, 1 + few + 2048), bp, 1200)
    g = pv.RFI(bp, cr=5.0, sr=4.0, history=1200)
    d = torch.from_numpy(data).to(cuda)
    for n, want in ((1, 1), (few, 1), (few + 1, 5), (2048 + few, 6)):
        before = pv.launches()
        g.run(d[:n])
        assert pv.launches() - before == want


@pytest.mark.parametrize("nsub,nchan,kind", [
    (8, 16, "rejected"), (8, 16, "zeros"), (8, 16, "terms"), (320, 16, "rejected"), (513, 16, "rejected"),
    (513, 16, "zeros"), (513, 16, "terms"), (128, 16, "terms"), (1025, 16, "rejected"), (8, 16, "burst"),
])
def test_blocks_left_to_the_walk(pv, oracle, cuda, nsub, nchan, kind):
    """Spectra that a scan does over one by one, most of a block's: it leaves
    the rest to the walk, from the block's start, its middle, and not at all
    where the rest is quiet; the blocks after it go on from there."""
    rng = np.random.default_rng(nsub + len(kind))
    nbins, H = nsub * nchan, 1100
    nt = H + 3000
    data = stokes_filterbank(rng, nt, nsub, nchan)
    bp = make_bp_text(nbins, START, WIDTH, 1000.0, 50.0, (0.3,) if kind == "terms" else ())
    if kind == "rejected":  # two calls are left to the walk; quiet; then every third
        data[H + 300:H + 1450] *= 2.0
        data[H + 1900::3] *= 2.0
    elif kind == "burst":  # 70 spectra, then quiet
        data[H + 300:H + 370] *= 2.0
    elif kind == "zeros":
        data[:H + 900] = 0.0
    _run(pv, oracle, cuda, data, (700, H + 100, H + 600, H + 1100, H + 1600, H + 2600), bp, H)


def test_polarisations_of_blocks_left_to_the_walk(pv, oracle, cuda):
    import torch
    rng = np.random.default_rng(2)
    nt, nsub, npol, nchan = 2500, 8, 4, 16
    data = rng.normal(1000.0, 50.0, (nt, nsub, npol, nchan)).astype(np.float32)
    data[:, 3, 0, 5] *= 20.0
    data[1200:] *= 2.0
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0)
    kw = dict(cr=5.0, sr=4.0, history=1100, zero_dming=True)
    outs = []
    for split in (None, 0):  # in blocks, and walked throughout
        d = torch.from_numpy(data).to(cuda)
        r = pv.RFI(bp, split=split, **kw)
        f = [r.run(d[a:b], flags=True).cpu().numpy() for a, b in ((0, 1500), (1500, 2000), (2000, nt))]
        outs.append((d.cpu().numpy(), np.concatenate(f)))
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    assert (outs[0][1][1300:] & 2).all()


@pytest.mark.parametrize("nsub", [8, 128])
@pytest.mark.parametrize("terms", [(), (0.3,)])
def test_rms_of_each_spectrum(pv, oracle, cuda, nsub, terms):
    """Without computeRMSfromMean the RMS is each spectrum's own after
    flattening, and the spectra are walked, one launch a call."""
    import torch
    nt, nchan = 2600, 16
    data = stokes_filterbank(np.random.default_rng(nsub), nt, nsub, nchan)
    bp = make_bp_text(nsub * nchan, START, WIDTH, 1000.0, 50.0, terms)
    kw = dict(cr=5.0, sr=4.0, history=1100, zero_dming=True, mean_over_rms=False)
    g = pv.RFI(bp, **kw)
    o = oracle.RFI(bp, mode=1, parts=pv.load().pv_rfi_parts(nsub * nchan), **kw)
    for a, b in ((0, 1), (1, 1500), (1500, nt)):
        d = np.ascontiguousarray(data[a:b])
        dd = torch.from_numpy(d).to(cuda)
        before = pv.launches()
        gf = g.run(dd, flags=True).cpu().numpy()
        assert pv.launches() - before == 1
        assert np.array_equal(gf, o.run(d, flags=True))
        assert np.array_equal(dd.cpu().numpy(), d)
