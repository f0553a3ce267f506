"""The as-of join of two sides in time order (merged, without a sort) against
a search over the sorted build side, which the same join takes for probe rows
in another order: steps and slices with remainders, equal times, chains of one
slot inside a step, NULL and unknown keys, tolerances, every key form."""
import numpy as np
import pytest

import oracle as O
import qeg
from util import to_gpu

pytestmark = pytest.mark.gpu


def expected(bkey, bts, pkey, pts, tol):
    """Build row of every probe row, -1: none (stable order of equal times)."""
    big = 1 << 40
    comp = bkey * big + bts
    order = np.argsort(comp, kind="stable")
    at = np.searchsorted(comp[order], pkey * big + pts, side="right") - 1
    row = order[np.maximum(at, 0)]
    ok = (at >= 0) & (pkey >= 0)
    ok &= bkey[row] == pkey
    if tol is not None:
        ok &= pts - bts[row] <= tol
    return np.where(ok, row, -1)


def run(ctx, build, probe, nkeys, join_type, tol, batches=1):
    j = qeg.AsofJoin(ctx, [c.type for c in probe], [c.type for c in build], list(range(nkeys)), list(range(nkeys)),
                     nkeys, nkeys, join_type, tol)
    try:
        bcols = [to_gpu(c) for c in build]
        j.build(bcols)
        j.build_finish()
        brow = []
        n = probe[0].n
        cut = [n * i // batches for i in range(batches + 1)]
        for a, b in zip(cut[:-1], cut[1:]):
            pcols = [to_gpu(O.TCol(c.type, c.values[a:b], None if c.valid is None else c.valid[a:b])) for c in probe]
            m = j.probe(pcols)
            if not m:
                continue
            cols = j.fetch(0, m)
            v, ok = cols[-1]
            brow.append(np.where(ok != 0, v, -1))
        return np.concatenate(brow) if brow else np.zeros(0, np.int64)
    finally:
        j.close()


# Key forms: a dense I32 key (plain rows), with NULLs, a dense I64 key, a
# hashed key, two keys; times as TS or I32.
@pytest.mark.parametrize("form", ["i32", "i32_null", "i64", "hashed", "two"])
@pytest.mark.parametrize("nb,npr,nsym", [(128, 128, 40), (129, 1000, 100), (5000, 4999, 60), (20000, 70001, 700),
                                         (40000, 50000, 16000), (30000, 30000, 3), (3000, 3000, 20000)])
@pytest.mark.parametrize("join_type,tol", [(O.LEFT, None), (O.INNER, 3000)])
def test_merge(ctx, form, nb, npr, nsym, join_type, tol):
    rng = np.random.default_rng(nb + nsym)
    span = 1 << 20
    wide = form != "i64"
    # A slow clock (equal times within and between the sides), both sides in order.
    bts = np.sort(rng.integers(100, span, nb) // 64 * 64)
    pts = np.sort(rng.integers(0, span + 500, npr) // 32 * 32)
    draw = lambda n: np.minimum((nsym ** rng.random(n)).astype(np.int64) - 1, nsym - 1)  # skewed
    bkey, pkey = draw(nb), draw(npr)
    pkey[rng.random(npr) < 0.05] = nsym + 5  # unknown
    bok = np.ones(nb, bool)
    pok = np.ones(npr, bool)
    if form == "i32_null":
        bok, pok = rng.random(nb) > 0.1, rng.random(npr) > 0.1
    ts = (lambda v: O.TCol(O.TS, v.astype(np.int64))) if wide else (lambda v: O.TCol(O.I32, v.astype(np.int32)))

    def keys(k, ok):
        if form == "i64":
            return [O.TCol(O.I64, k - 7)]
        if form == "hashed":
            return [O.TCol(O.I64, k * 0x51ED270B7 + 3)]
        if form == "two":
            return [O.TCol(O.I32, (k % 11).astype(np.int32)), O.TCol(O.I64, k // 11)]
        return [O.TCol(O.I32, k.astype(np.int32), None if ok.all() else ok)]

    nkeys = 2 if form == "two" else 1
    build = keys(bkey, bok) + [ts(bts), O.TCol(O.I64, np.arange(nb))]
    probe = keys(pkey, pok) + [ts(pts), O.TCol(O.I64, np.arange(npr))]
    exp = expected(np.where(bok, bkey, nsym + 77), bts, np.where(pok, pkey, -1), pts, tol)
    want = np.arange(npr) if join_type == O.LEFT else np.flatnonzero(exp >= 0)
    for batches in (1, 3):  # three batches: smaller than some of the build sides
        assert np.array_equal(run(ctx, build, probe, nkeys, join_type, tol, batches), exp[want])
    # The same rows in another order: noticed, and answered from sorted runs.
    perm = rng.permutation(npr)
    shuffled = [O.TCol(c.type, c.values[perm], None if c.valid is None else c.valid[perm]) for c in probe]
    brow = run(ctx, build, shuffled, nkeys, join_type, tol)
    e = exp[perm]
    assert np.array_equal(brow, e if join_type == O.LEFT else e[e >= 0])
    # One neighbouring pair out of order, somewhere.
    steps = np.flatnonzero(np.diff(pts) > 0)
    at = int(steps[len(steps) // 5])
    perm = np.arange(npr)
    perm[[at, at + 1]] = [at + 1, at]
    swapped = [O.TCol(c.type, c.values[perm], None if c.valid is None else c.valid[perm]) for c in probe]
    brow = run(ctx, build, swapped, nkeys, join_type, tol)
    e = exp[perm]
    assert np.array_equal(brow, e if join_type == O.LEFT else e[e >= 0])
