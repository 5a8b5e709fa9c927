"""The pipelined dedispersion's tiles on linear and ring rows against the
oracle's FP32 sums, bit for bit: sizes around each tile's edges, delay spreads
that only some tiles hold, rows at any stride, buffers at any alignment, and
rows that end inside the spans (zeros beyond row_len, the next row where rows
are contiguous, zeros beyond the buffer)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # nchan, tdms, nout, fch1, foff, DM step over tsamp
    (40, 9, 255, 150.0, -0.05, 400.0),     # 8 x 256
    (33, 17, 1025, 150.0, -0.05, 400.0),
    (70, 300, 5003, 150.0, -0.05, 300.0),
    (50, 600, 16500, 150.0, -0.05, 50.0),  # 16 x 1024
    (24, 512, 10976, 150.0, -0.05, 100.0),  # 8 x 1024
    (90, 40, 3000, 115.0, -0.05, 30000.0),  # spreads of thousands of samples
]


def _case(pv, oracle, case, seed=0):
    nchan, tdms, nout, fch1, foff, step = case
    k, _ = pv.dm_shifts(fch1, foff, nchan)
    start, step = np.float32(1.5), np.float32(step)
    ms = int(oracle.shift_table(k, tdms, start, step).max())
    return k, start, step, ms, np.random.default_rng(seed + nchan)


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("extra", [0, 1, 2, 3])
def test_linear_rows(pv, oracle, cuda, case, extra):
    import torch
    nchan, tdms, nout = case[:3]
    k, start, step, ms, rng = _case(pv, oracle, case)
    width = nout + ms + extra  # extra 0: the last channel's last sample is the buffer's last
    x = rng.standard_normal((nchan, width)).astype(np.float32)
    want = oracle.dedisperse(x, nout, tdms, k, start, step)
    kd = torch.from_numpy(k).to(cuda)
    got = pv.dedisperse(torch.from_numpy(x).to(cuda), nout, tdms, kd, float(start), float(step))
    assert np.array_equal(got.cpu().numpy(), want)
    plan = pv.DedispPlan(k, tdms, float(start), float(step))
    assert np.array_equal(plan.run(torch.from_numpy(x).to(cuda), nout).cpu().numpy(), want)
    assert plan.status() == 0
    if extra == 1:  # a buffer that is not 16-byte aligned
        flat = torch.zeros(nchan * width + 1, device=cuda)
        flat[1:] = torch.from_numpy(x.reshape(-1)).to(cuda)
        got = pv.dedisperse(flat[1:].view(nchan, width), nout, tdms, kd, float(start), float(step))
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("case", CASES[:3] + CASES[5:])
@pytest.mark.parametrize("short", [1, 700])
def test_rows_that_end_early(pv, oracle, cuda, case, short):
    """row_len below what the delays reach: zeros beyond it; the same of a
    contiguous buffer: the next row, and zeros beyond the last."""
    import torch
    nchan, tdms, nout = case[:3]
    k, start, step, ms, rng = _case(pv, oracle, case, 1)
    length = max(nout + ms - short, 1)
    x = rng.standard_normal((nchan, length + 5)).astype(np.float32)
    full = np.zeros((nchan, nout + ms + 1), np.float32)
    full[:, :length] = x[:, :length]
    want = oracle.dedisperse(full, nout, tdms, k, start, step)
    kd = torch.from_numpy(k).to(cuda)
    got = pv.dedisperse(torch.from_numpy(x).to(cuda), nout, tdms, kd, float(start), float(step), row_len=length)
    assert np.array_equal(got.cpu().numpy(), want)
    y = np.ascontiguousarray(x[:, :length])
    flat = np.concatenate([y.reshape(-1), np.zeros(nout + ms + 1, np.float32)])
    for c in range(nchan):
        full[c] = flat[c * length:c * length + nout + ms + 1]
    want = oracle.dedisperse(full, nout, tdms, k, start, step)
    got = pv.dedisperse(torch.from_numpy(y).to(cuda), nout, tdms, kd, float(start), float(step))
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("case", CASES)
def test_ring_rows(pv, oracle, cuda, case):
    import torch
    nchan, tdms, nout = case[:3]
    k, start, step, ms, rng = _case(pv, oracle, case, 2)
    ring = (nout + ms + 1100 + 3) // 4 * 4
    lin = rng.standard_normal((nchan, ring)).astype(np.float32)
    want = oracle.dedisperse(lin, nout, tdms, k, start, step)
    plan = pv.DedispPlan(k, tdms, float(start), float(step))
    for base in (0, ring - 5):
        x = np.roll(lin, base, axis=1)
        got = plan.run(torch.from_numpy(np.ascontiguousarray(x)).to(cuda), nout, ring_len=ring, t_base=base)
        assert np.array_equal(got.cpu().numpy(), want)
    assert plan.status() == 0


PAIR_CASES = [
    # Trial pairs, delay differences of 0 to 28 samples (from 16 on each
    # trial reads its own words): rows enough to fill every SM.  14 x 1056
    # on a grid of one and of two trials more than its tiles, 8 x 1056 on an odd one; a last
    # sample tile of one sample and one that is full.
    (9, 1024, 8449, 150.0, -0.05, 30.0),
    (17, 1023, 8448, 150.0, -0.05, 5000.0),
    (17, 1024, 8448, 150.0, -0.05, 14000.0),
    (20, 513, 10976, 150.0, -0.05, 4600.0),
    (3, 4097, 9000, 1300.0, -0.04, 0.0),
]


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("case", PAIR_CASES)
def test_trial_pairs(pv, oracle, cuda, case, ring):
    import torch
    nchan, tdms, nout = case[:3]
    k, start, step, ms, rng = _case(pv, oracle, case, 3)
    width = nout + ms + (1100 if ring else 1)
    width = (width + 3) // 4 * 4 if ring else width
    x = rng.standard_normal((nchan, width)).astype(np.float32)
    want = oracle.dedisperse(x, nout, tdms, k, start, step)
    plan = pv.DedispPlan(k, tdms, float(start), float(step))
    base = width - 7 if ring else 0
    xd = torch.from_numpy(np.ascontiguousarray(np.roll(x, base, axis=1))).to(cuda)
    got = plan.run(xd, nout, ring_len=width if ring else 0, t_base=base)
    assert np.array_equal(got.cpu().numpy(), want)
    assert plan.status() == 0


NARROW_CASES = [
    # few trials or samples, or delays far apart from one trial to the next (2.4e-4 per unit of
    # the step and channel at the lowest): 8 x 256 and 4 x 256 in 32-channel stages, 4, 2 and
    # 1 x 1024, 1 x 256; fewer trials than the eight that the rule's spread is taken of
    (70, 512, 1025, 150.0, -0.05, 600.0),
    (65, 99, 3000, 150.0, -0.05, 5.0),
    (33, 64, 513, 150.0, -0.05, 5000.0),
    (33, 200, 3000, 150.0, -0.05, 40000.0),
    (31, 61, 9001, 150.0, -0.05, 190000.0),
    (33, 16, 16001, 150.0, -0.05, 500000.0),
    (40, 20, 1000, 150.0, -0.05, 1000000.0),
    (33, 7, 300, 150.0, -0.05, 5000.0),
    (5, 1, 255, 150.0, -0.05, 5000.0),
]


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("case", NARROW_CASES)
def test_narrow_tiles(pv, oracle, cuda, case, ring):
    test_trial_pairs(pv, oracle, cuda, case, ring)


@pytest.mark.parametrize("case", NARROW_CASES[1:7])
def test_narrow_tiles_past_the_rows_end(pv, oracle, cuda, case):
    test_rows_that_end_early(pv, oracle, cuda, case, 700)


def test_short_ring_stays_refused(pv, cuda):
    """A ring shorter than a wide tile's span is an error whichever tile would be faster."""
    import torch
    k, _ = pv.dm_shifts(150.0, -0.05, 33)
    plan = pv.DedispPlan(k, 64, 0.0, 20000.0)
    x = torch.zeros(33, 1600, device=cuda)
    with pytest.raises(Exception):
        plan.run(x, 1000, ring_len=1600)


TILES = [
    # (trials, samples, channels per stage) of each tile on 152 SMs, zeros for the plain kernel; one
    # trial and one sample more than whole tiles
    ((0, 0, 0), (4, 1009, 9001, 150.0, -0.05, 30.0)),
    ((16, 1024, 8), (24, 513, 10241, 150.0, -0.05, 100.0)),
    ((16, 1024, 2), (90, 65, 20481, 150.0, -0.1, 10000.0)),
    ((8, 1024, 8), (33, 161, 18433, 150.0, -0.05, 3089.0)),
    ((8, 256, 16), (70, 297, 5121, 150.0, -0.05, 300.0)),
    ((14, 1056, 8), (200, 169, 21121, 150.0, -0.05, 763.0)),
    ((8, 1056, 8), (300, 257, 10561, 150.0, -0.1, 4.0)),
    ((8, 256, 32), (128, 153, 3329, 150.0, -0.05, 4745.0)),
    ((4, 256, 32), (65, 101, 3073, 150.0, -0.05, 5.0)),
    ((4, 1024, 8), (200, 73, 15361, 150.0, -0.05, 54.0)),
    ((2, 1024, 8), (90, 39, 11265, 150.0, -0.05, 18853.0)),
    ((1, 1024, 8), (70, 8, 29697, 150.0, -0.1, 21752.0)),
    ((1, 256, 32), (70, 7, 3585, 150.0, -0.1, 166.0)),
]


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("tile,case", TILES)
def test_every_tile(pv, oracle, cuda, tile, case, ring):
    """Each tile on sizes that the rule gives it, so that a change of the rule
    cannot leave one untested."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the tiles of 152 SMs")
    k, start, step, ms, _ = _case(pv, oracle, case)
    plan = pv.DedispPlan(k, case[1], float(start), float(step))
    assert plan.tile(case[2], (case[2] + ms + 1100 + 3) // 4 * 4 if ring else 0) == tile
    test_trial_pairs(pv, oracle, cuda, case, ring)


@pytest.mark.parametrize("nchan", [1, 2, 4, 5, 8, 32])
def test_few_channels_take_no_trial_pairs(pv, oracle, cuda, nchan):
    """A pair's stores cost what 64 channels do (1024 trials x 16384 samples of
    one channel: 83 us against 17 by the plain kernel)."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the tiles of 152 SMs")
    k, _ = pv.dm_shifts(150.0, -0.05, nchan)
    plan = pv.DedispPlan(k, 1024, 0.0, 1.0)
    for ring in (0, 18000):
        assert plan.tile(16384, ring) == ((0, 0, 0) if nchan <= 4 else (16, 1024, 8))
