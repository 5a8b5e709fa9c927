"""The two-phase Stokes-I channeliser (16, 32 and 64 channels) against the
any-shape kernel, bit for bit, over two calls that carry the tap history:
blocks around the phase (8), the stream (32 to 256) and the CTA's streams,
every window it takes, int16 and complex float voltages, and buffers that
16-byte accesses do not fit (another kernel's)."""
import numpy as np
import pytest

from gen import voltages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan", [16, 32, 64])
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


@pytest.mark.parametrize("nchan", [16, 32, 64])
@pytest.mark.parametrize("window,chunk", [(4, 2), (1, 9), (8, 70)])
def test_packets_equal_voltages(pv, cuda, nchan, window, chunk):
    """Chunks read from LOFAR packets in place, two in a row, against the same
    voltages: the filterbank of a packet-fed beam."""
    import torch
    rng = np.random.default_rng(nchan * window + chunk)
    nsub, per, n = 6, 3, chunk * window * nchan
    kw = dict(nsub=nsub, nchan_sub=nchan, int_time=window, fch1=150.0, foff=-0.01, tsamp=1e-3, tdms=2, dm_step=0.01,
              chunk=chunk, rfi_active=0, bin_pow2=0, prefilled=1)
    a = pv.Beam(pv.beam_config(**kw))
    b = pv.Beam(pv.beam_config(**kw, udp_packet_bytes=16 + per * 128, udp_subbands=per))
    for _ in range(2):
        v, _ = voltages(rng, nsub, 2, n)
        body = v.reshape(nsub // per, per, 2, n // 16, 16, 2).transpose(0, 3, 1, 4, 2, 5)
        pk = np.zeros((nsub // per, n // 16, 16 + per * 128), np.uint8)
        pk[:, :, 16:] = np.ascontiguousarray(body).view(np.uint8).reshape(nsub // per, n // 16, -1)
        a.process(torch.from_numpy(v.reshape(nsub, 2, -1)).to(cuda))
        b.process(torch.from_numpy(pk.reshape(-1)).to(cuda))
        fa, fb = (pv.device_array(x.buffers()[0], (chunk, nsub, 1, nchan)).cpu().numpy() for x in (a, b))
        assert np.array_equal(fa, fb) and fa.any()
