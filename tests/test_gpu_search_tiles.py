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


def test_noalloc_calls_that_overlapped_leave_the_next_one_right(pv, oracle, cuda):
    """Calls of pv_analyse_noalloc that overlap on the GPU spoil their own
    results; the calls after them are right again."""
    import ctypes as C
    import threading
    import torch
    L = pv.load()
    L.pv_analyse_noalloc.restype = C.c_int
    L.pv_analyse_noalloc.argtypes = L.pv_analyse.argtypes
    shapes = [(1024, 8192, 3), (700, 8192, 3)]
    data = [torch.zeros(t, n, device=cuda) for t, n, _ in shapes]
    lists = [torch.zeros(4 << 12, dtype=torch.int32, device=cuda) for _ in shapes]
    streams = [torch.cuda.Stream() for _ in shapes]
    torch.cuda.synchronize()
    gate = threading.Barrier(2)
    bad = []

    def calls(i):
        t, n, p = shapes[i]
        total = C.c_longlong()
        gate.wait()
        for _ in range(200):
            if L.pv_analyse_noalloc(data[i].data_ptr(), n, t, n, 5.0, 1.0, p, lists[i].data_ptr(), 1 << 12,
                                    C.byref(total), streams[i].cuda_stream):
                bad.append(i)

    threads = [threading.Thread(target=calls, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not bad
    rng = np.random.default_rng(3)
    for _ in range(3):
        x = rng.standard_normal((64, 4096)).astype(np.float32)
        want = oracle.analyse(x, 2.6, 1.0, 6)
        d = torch.from_numpy(x).to(cuda)
        ev = torch.zeros(4 * len(want), dtype=torch.int32, device=cuda)
        total = C.c_longlong()
        pv.check(L.pv_analyse_noalloc(d.data_ptr(), 4096, 64, 4096, 2.6, 1.0, 6, ev.data_ptr(), len(want),
                                      C.byref(total), torch.cuda.current_stream().cuda_stream))
        assert total.value == len(want)
        assert np.array_equal(ev.cpu().numpy().view(pv.EVENT_DTYPE), want.astype(pv.EVENT_DTYPE))
