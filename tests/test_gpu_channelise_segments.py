"""The two-phase Stokes-I channeliser (16 and 32 channels) against the
any-shape kernel, bit for bit, over two calls that carry the tap history:
blocks around the phase (8), the stream (32 to 256) and the CTA's streams,
every window it takes, int16 and complex float voltages, and buffers that
16-byte accesses do not fit (another kernel's)."""
import numpy as np
import pytest

from gen import voltages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan", [16, 32])
@pytest.mark.parametrize("window,nblk", [(1, 7), (4, 8), (2, 9), (8, 255), (4, 257), (8, 263), (4, 511), (1, 1030),
                                         (4, 2049), (16, 300)])
@pytest.mark.parametrize("int16", [True, False])
def test_segments_equal_the_any_shape_kernel(pv, oracle, cuda, monkeypatch, nchan, window, nblk, int16):
    import torch
    rng = np.random.default_rng(nchan + nblk)
    nsub = 3
    v16, x = voltages(rng, nsub, 2, nblk * nchan)
    coeffs = oracle.fir_coefficients(8, nchan, "kaiser").astype(np.float32)
    host = v16.reshape(nsub, 2, -1) if int16 else x
    d_in = torch.from_numpy(host).to(cuda)
    flat = torch.zeros(d_in.numel() + 1, dtype=d_in.dtype, device=cuda)
    flat[1:] = d_in.reshape(-1)
    outs = {}
    for mode in ("segments", "unaligned", "any"):
        if mode == "any":
            monkeypatch.setenv("PV_CHAN_GENERIC", "1")
        f = pv.PPF(nchan, 8, coeffs=coeffs)
        src = flat[1:].view(d_in.shape) if mode == "unaligned" and not int16 else d_in
        outs[mode] = [f.channelise(src, 1, window, 1).cpu().numpy() for _ in range(2)]
    for a, b, c in zip(outs["segments"], outs["unaligned"], outs["any"]):
        assert a.shape == (nblk // min(window, nblk), nsub, 1, nchan)
        assert np.array_equal(a, c) and np.array_equal(b, c)
