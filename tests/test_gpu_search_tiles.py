"""The search in tiles of 128 (trial, block) pairs against the oracle, event by
event: tiles that span rows, rows of fewer blocks than a tile, the last tile
partly filled, every block size, rows that 16-byte reads do not fit, windows
where every sample is an event (a tile's events in order, the total beyond the
list's end) and none is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pow2", range(9))
@pytest.mark.parametrize("tdms,nsamp", [(3, 4099), (300, 517), (129, 256), (1, 33000)])
def test_events_of_every_block_size(pv, oracle, cuda, pow2, tdms, nsamp):
    import torch
    rng = np.random.default_rng(pow2 * 1000 + tdms)
    for width in (nsamp, (nsamp + 3) // 4 * 4):  # rows at any alignment, and rows of whole 16 bytes
        x = rng.standard_normal((tdms, width)).astype(np.float32)
        x[tdms // 2, width // 3:width // 3 + 20] += 5.0
        want = oracle.analyse(x[:, :width], 2.6, 1.0, pow2)
        got, n = pv.analyse(torch.from_numpy(x).to(cuda), 2.6, 1.0, pow2)
        assert n == len(want) and np.array_equal(got, want.astype(got.dtype))


def test_every_sample_an_event_and_a_short_list(pv, oracle, cuda):
    import torch
    x = np.ones((40, 1024), np.float32)
    want = oracle.analyse(x, 0.5, 1.0, 6)
    d = torch.from_numpy(x).to(cuda)
    got, n = pv.analyse(d, 0.5, 1.0, 6)
    assert n == len(want) == 1 + 40 * sum(1024 >> k for k in range(7)) and np.array_equal(got, want.astype(got.dtype))
    got, n = pv.analyse(d, 0.5, 1.0, 6, cap=1000)
    assert n == len(want) and np.array_equal(got, want.astype(got.dtype)[:1000])
    got, n = pv.analyse(torch.from_numpy(-x).to(cuda), 0.5, 1.0, 6)
    assert n == 1
