"""GROUP BY results fetched into host and device buffers: row ranges at word
and block edges, small results (one page-locked hop) and large ones (copies),
aligned and unaligned device destinations. Every key is its own group, so the
expected cells are the input's (the reference's Aggregate::next emits the same
cells, ops/aggregate.cpp:439-493)."""
import ctypes

import numpy as np
import pytest

import qeg

pytestmark = pytest.mark.gpu


def finished(ctx, n):
    """An aggregate over n distinct keys: MAX of a BOOL, an I32 and an F64
    column, the last two with NULLs (multiples of 7 and of 5)."""
    key = np.arange(n, dtype=np.int64) * 3 + 1
    b = (np.arange(n) % 2).astype(np.uint8)
    i = (np.arange(n) * 11 - 5).astype(np.int32)
    f = np.arange(n) * 0.5 - 3.0
    iv, fv = np.arange(n) % 7 != 0, np.arange(n) % 5 != 0
    a = qeg.Aggregate(ctx, [qeg.I64, qeg.BOOL, qeg.I32, qeg.F64], [0], [(qeg.MAX, 1), (qeg.MAX, 2), (qeg.MAX, 3)])
    a.consume([qeg.Col(key), qeg.Col(b, None, qeg.BOOL), qeg.Col(i, qeg.pack_validity(iv)),
               qeg.Col(f, qeg.pack_validity(fv))])
    assert a.finish() == n
    return a, [(b, np.ones(n, bool)), (i, iv), (f, fv)]


def check(keys, key_ok, cols, want):
    row = (np.asarray(keys) - 1) // 3
    assert bool(np.all(key_ok))
    for (v, ok), (wv, wok) in zip(cols, want):
        assert np.array_equal(ok, wok[row])
        assert np.array_equal(np.asarray(v)[ok], wv[row][ok])
    return row


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1023, 1025, 12_000, 150_001])
def test_fetch_ranges_to_host(ctx, n):
    a, want = finished(ctx, n)
    seen = []
    cuts = sorted({0, min(1, n), min(65, n), n // 2, n})  # odd starts: unaligned sources
    for lo, hi in zip(cuts[:-1], cuts[1:]):
        res = a.fetch(lo, hi - lo)
        seen.append(check(*res[0], res[1:], want))
    assert np.array_equal(np.sort(np.concatenate(seen)), np.arange(n))
    a.close()


@pytest.mark.parametrize("shift", [0, 1, 4, 8])
@pytest.mark.parametrize("n", [1, 65, 5000])
def test_fetch_to_device_at_any_alignment(ctx, n, shift):
    torch = pytest.importorskip("torch")
    a, want = finished(ctx, n)
    dt = [np.int64, np.uint8, np.int32, np.float64]
    nw = (n + 63) // 64
    bufs = [(torch.full((n * 8 + 64,), 0xA5, dtype=torch.uint8, device="cuda"),
             torch.full((nw * 8 + 64,), 0xA5, dtype=torch.uint8, device="cuda")) for _ in dt]
    torch.cuda.synchronize()
    outs = (qeg.OutColumn * 4)()
    flags = (ctypes.c_int32 * 4)()
    for c, (v, w) in enumerate(bufs):
        outs[c] = qeg.OutColumn(v.data_ptr() + shift, w.data_ptr() + shift, ctypes.addressof(flags) + 4 * c)
    assert qeg.lib().qeg_agg_fetch(a.p, 0, n, outs) == 0
    got = []
    for (v, w), d in zip(bufs, dt):
        hv, hw = v.cpu().numpy(), w.cpu().numpy()
        size = n * np.dtype(d).itemsize
        assert (hv[:shift] == 0xA5).all() and (hv[shift + size:] == 0xA5).all()  # nothing beyond the column
        assert (hw[:shift] == 0xA5).all() and (hw[shift + nw * 8:] == 0xA5).all()
        words = hw[shift:shift + nw * 8].copy().view(np.uint64)
        if n % 64:
            assert int(words[-1]) >> (n % 64) == (1 << (64 - n % 64)) - 1  # padding bits set
        got.append((hv[shift:shift + size].copy().view(d), qeg.unpack_validity(words, n)))
    check(*got[0], got[1:], want)
    assert list(flags) == [1, 1, 0, 0]
    a.close()
