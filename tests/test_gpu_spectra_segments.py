"""The complex spectra of 16 and 32 channels (the two-phase kernel) and of every
other channel count against the oracle, over two calls that carry the history,
and the integrator on values that 16-byte reads fit and do not."""
import numpy as np
import pytest

from gen import voltages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan", [1, 2, 4, 8, 16, 20, 32, 64, 128, 256])
@pytest.mark.parametrize("ntaps,nblk", [(8, 7), (8, 133), (5, 40), (8, 3)])
def test_spectra(pv, oracle, cuda, monkeypatch, nchan, ntaps, nblk):
    import torch
    rng = np.random.default_rng(nchan + nblk)
    nsub = 3
    _, x = voltages(rng, nsub, 2, nblk * nchan)
    coeffs = np.ones((8, 1), np.float32) if nchan == 1 else \
        oracle.fir_coefficients(ntaps, nchan, "kaiser").astype(np.float32)
    f, g = pv.PPF(nchan, ntaps, coeffs=coeffs), None
    o = oracle.PPF(nchan, 8 if nchan == 1 else ntaps, coeffs)
    d = torch.from_numpy(x).to(cuda)
    for _ in range(2):
        got = f.run(d).cpu().numpy()
        want = o.run(x.reshape(nsub, 2, nblk, nchan))
        scale = np.sqrt(np.mean(np.abs(want) ** 2))
        assert np.max(np.abs(got - want)) <= 2e-5 * scale * max(1.0, np.sqrt(nchan) / 4)
    if nchan in (16, 32) and ntaps == 8:  # bit for bit with the any-shape kernel
        outs = []
        for mode in (0, 1):
            if mode:
                monkeypatch.setenv("PV_CHAN_GENERIC", "1")
            g = pv.PPF(nchan, ntaps, coeffs=coeffs)
            outs.append([g.run(d).cpu().numpy() for _ in range(2)])
        for a, b in zip(*outs):
            assert np.array_equal(a, b)


def test_infinite_voltages(pv, oracle, cuda, monkeypatch):
    """An infinite sample makes the same values of a block infinite or NaN in
    both kernels."""
    import torch
    rng = np.random.default_rng(3)
    _, x = voltages(rng, 2, 2, 20 * 16)
    x[1, 0, 37] = np.inf
    d = torch.from_numpy(x).to(cuda)
    outs = []
    for mode in (0, 1):
        if mode:
            monkeypatch.setenv("PV_CHAN_GENERIC", "1")
        outs.append((pv.PPF(16, 8).run(d).cpu().numpy(), pv.PPF(16, 8).channelise(d, 1, 4, 1).cpu().numpy()))
    for a, b in zip(*outs):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("shape,window", [((37, 3, 4, 16), 16), ((9, 5, 1, 7), 2), ((40, 62, 4, 32), 7), ((5, 1, 1, 4), 9)])
def test_integrator(pv, oracle, cuda, shape, window):
    import torch
    x = np.random.default_rng(1).standard_normal(shape).astype(np.float32)
    want = oracle.integrate(x, window, 1)
    d = torch.from_numpy(x).to(cuda)
    assert np.array_equal(pv.integrate(d, window).cpu().numpy(), want)
    flat = torch.zeros(d.numel() + 1, device=cuda)
    flat[1:] = d.reshape(-1)
    assert np.array_equal(pv.integrate(flat[1:].view(shape), window).cpu().numpy(), want)


@pytest.mark.parametrize("nchan", [16, 64])
def test_more_subbands_than_a_grid_holds_are_refused(pv, cuda, nchan):
    """The limit of complex spectra is one of the entry point, not of a kernel."""
    import torch
    x = torch.zeros(65536, 2, 7 * nchan, dtype=torch.complex64, device=cuda)
    with pytest.raises(pv.PvError, match="too many subbands"):
        pv.PPF(nchan, 8).run(x)
    assert pv.PPF(nchan, 8).run(x[:65535]).shape[1] == 65535
