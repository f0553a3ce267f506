"""Materialised joins against the oracle at the edges of the output path:
chunk and word remainders, unique and repeated build keys, one, two and three
key columns, dense and hashed tables, packed build rows of 32 and 64 bytes and
rows too wide to pack, results fetched whole, in unaligned ranges, into device
and host buffers."""
import numpy as np
import pytest

import oracle as O
import qeg
from util import to_gpu

pytestmark = pytest.mark.gpu


def check(types, got, exp):
    grows = list(zip(*[[None if not ok else (float(x) if t == O.F64 else int(x)) for x, ok in zip(v.tolist(), k.tolist())]
                       for t, (v, k) in zip(types, got)]))
    m = O.compare(types, grows, types, exp)
    assert m is None, m


def build_keys(rng, nb, kind, dup):
    ids = rng.permutation(nb) // dup
    return ids if kind == "dense" else ids * 0x51ED270B7 + 3


def columns(rng, n, nkeys, ids, null_pct):
    ok = lambda: rng.random(n) >= null_pct / 100.0 if null_pct else None
    keys = [O.TCol(O.I64, ids.astype(np.int64), ok())]
    if nkeys > 1:
        keys.append(O.TCol(O.I32, (ids % 7).astype(np.int32)))
    if nkeys > 2:
        keys.append(O.TCol(O.BOOL, (ids % 2).astype(np.uint8)))
    return keys


WIDTHS = {"narrow": [O.F64, O.I32], "wide": [O.F64, O.I64, O.TS, O.I32, O.BOOL],
          "widest": [O.I64] * 8}  # 32-byte rows, 64-byte rows, not packed


def payload(rng, n, types):
    out = []
    for i, t in enumerate(types):
        v = {O.F64: rng.normal(0, 9, n), O.I32: rng.integers(-99, 99, n).astype(np.int32),
             O.BOOL: rng.integers(0, 2, n).astype(np.uint8)}.get(t, rng.integers(-(1 << 50), 1 << 50, n))
        out.append(O.TCol(t, v, rng.random(n) > 0.2 if i % 2 == 0 else None))
    return out


@pytest.mark.parametrize("np_rows", [1, 127, 129, 4097])
@pytest.mark.parametrize("join_type", [O.INNER, O.LEFT])
@pytest.mark.parametrize("kind,nkeys", [("dense", 1), ("sparse", 1), ("sparse", 2), ("sparse", 3)])
@pytest.mark.parametrize("dup", [1, 3])
def test_join_rows(ctx, np_rows, join_type, kind, nkeys, dup):
    rng = np.random.default_rng(np_rows + 7 * nkeys + dup)
    nb = 1500
    bids = build_keys(rng, nb, kind, dup)
    hit = rng.random(np_rows) < 0.6
    pids = np.where(hit, bids[rng.integers(0, nb, np_rows)], rng.integers(-(1 << 40), 1 << 40, np_rows))
    build = columns(rng, nb, nkeys, bids, 3) + payload(rng, nb, WIDTHS["narrow"])
    probe = columns(rng, np_rows, nkeys, pids, 3) + payload(rng, np_rows, [O.I64])
    on = list(range(nkeys))
    et, erows = O.join(probe, build, on, on, join_type)
    j = qeg.Join(ctx, [c.type for c in probe], [c.type for c in build], on, on, join_type)
    j.build([to_gpu(c) for c in build])
    j.build_finish()
    pcols = [to_gpu(c) for c in probe]
    n = j.probe(pcols)
    try:
        check(et, j.fetch(), erows)
        if n > 70:  # an unaligned range and the rest
            a, b = j.fetch(0, 67), j.fetch(67, n - 67)
            check(et, [(np.concatenate([x[0], y[0]]), np.concatenate([x[1], y[1]])) for x, y in zip(a, b)], erows)
    finally:
        j.close()


@pytest.mark.parametrize("width", sorted(WIDTHS))
@pytest.mark.parametrize("join_type", [O.INNER, O.LEFT])
def test_join_rows_packed(ctx, width, join_type):
    """Enough output rows for the packed build rows; device and host outputs
    give the same cells as the input's own rows."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(len(width))
    nb, n = 60_000, 150_001
    bids = build_keys(rng, nb, "sparse", 1)
    row = rng.integers(0, nb, n)
    hit = rng.random(n) < 0.5
    pids = np.where(hit, bids[row], -1 - np.arange(n))
    bcols = payload(rng, nb, WIDTHS[width])
    build = [O.TCol(O.I64, bids.astype(np.int64))] + bcols
    probe = [O.TCol(O.I64, pids.astype(np.int64)), O.TCol(O.I32, np.arange(n, dtype=np.int32), rng.random(n) > 0.1)]
    j = qeg.Join(ctx, [c.type for c in probe], [c.type for c in build], [0], [0], join_type)
    j.build([to_gpu(c) for c in build])
    j.build_finish()
    pcols = [to_gpu(c, device=True) for c in probe]  # read in place until the last fetch
    out = j.probe(pcols)
    keep = np.ones(n, bool) if join_type == O.LEFT else hit
    assert out == keep.sum()

    def same(got, lo, hi):
        sel = np.nonzero(keep)[0][lo:hi]
        want = [(c.values[sel], np.ones(len(sel), bool) if c.valid is None else c.valid[sel]) for c in probe]
        want += [(c.values[row[sel]], hit[sel] if c.valid is None else hit[sel] & c.valid[row[sel]]) for c in build]
        for (v, ok), (wv, wok) in zip(got, want):
            assert np.array_equal(ok, wok)
            assert np.array_equal(np.asarray(v)[ok], wv[wok])

    try:
        same(j.fetch(), 0, out)
        for lo, hi in ((0, out), (64, out - 1), (65, 30_000)):
            dev = j.fetch_device(lo, hi - lo)
            same([(v.cpu().numpy()[:hi - lo], qeg.unpack_validity(w.cpu().numpy().view(np.uint64), hi - lo))
                  for v, w in dev], lo, hi)
    finally:
        j.close()
    del pcols
