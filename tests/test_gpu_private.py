"""Single-key GROUP BY through CTA-private tables, and two 4-byte keys packed
into one key word, against the oracle: few groups (rows of a warp on one slot),
more groups than a private table holds, keys clustered in time (the table is
flushed and refilled), NULL keys and key word 0, selections, small tables and
blocks, a global table that must grow, and batches that end the packing."""
import numpy as np
import pytest

import oracle as O
import qeg
from util import StrCanon, assert_same, gpu_rows, to_gpu

pytestmark = pytest.mark.gpu

INT_F64 = [(O.COUNT_STAR, 0), (O.SUM, 1), (O.SUM, 2), (O.MIN, 1), (O.MAX, 1)]
F64 = [(O.COUNT_STAR, 0), (O.SUM, 2), (O.AVG, 2), (O.MIN, 2), (O.MAX, 2)]
BARS = [(O.COUNT_STAR, 0), (O.SUM, 1), (O.MIN, 2), (O.MAX, 2), (O.AVG, 2)]
WIDE = [(O.COUNT, 1), (O.SUM, 1), (O.MIN, 1), (O.MAX, 1), (O.COUNT, 2), (O.AVG, 2), (O.MIN, 2), (O.MAX, 2),
        (O.SUM, 3), (O.MIN, 3)]


def run(ctx, batches, keys, aggs, config=None, sel=None, canon=None):
    a = qeg.Aggregate(ctx, [c.type for c in batches[0]], keys, aggs, config)
    for cols in batches:
        a.consume([to_gpu(c, canon) for c in cols], sel)
    a.finish()
    res = a.fetch()
    types = a.result_types
    a.close()
    return gpu_rows(res, types, canon)


def table(rng, key, nulls):
    n = len(key)
    ok = (lambda p: rng.random(n) >= p) if nulls else (lambda p: None)
    return [O.TCol(O.I64, key, ok(0.03)), O.TCol(O.I64, rng.integers(-(1 << 40), 1 << 40, n), None),
            O.TCol(O.F64, rng.normal(0, 1e3, n), ok(0.1)), O.TCol(O.I32, rng.integers(-9, 9, n).astype(np.int32), ok(0.5))]


def keys_of(rng, shape, n):
    if shape == "one":
        return np.full(n, 7, np.int64)
    if shape == "few":  # key word 0 among them
        return rng.integers(0, 5, n).astype(np.int64)
    if shape == "head":  # half of the rows on one key, the rest spread
        return np.where(rng.random(n) < 0.5, 11, rng.integers(0, 1 << 40, n) % 30_000).astype(np.int64)
    if shape == "many":
        return rng.integers(-(1 << 62), 1 << 62, n) // 3 % 40_000 - 20_000
    return np.arange(n, dtype=np.int64) // 40 * 16 + rng.integers(0, 16, n)  # clustered in time


@pytest.mark.parametrize("shape", ["one", "few", "head", "many", "time"])
@pytest.mark.parametrize("aggs,nulls", [(INT_F64, False), (INT_F64, True), (F64, False), (F64, True), (BARS, True),
                                        (WIDE, True), ([(O.COUNT_STAR, 0)], True)],
                         ids=["int_f64", "int_f64_nulls", "f64", "f64_nulls", "bars_nulls", "wide", "count"])
def test_private_tables(ctx, shape, aggs, nulls):
    rng = np.random.default_rng(len(shape) * 100 + len(aggs) * 2 + nulls)
    n = 300_007  # 74 CTAs of about 4,055 rows; every CTA's last warp is partial
    cols = table(rng, keys_of(rng, shape, n), nulls)
    ot, orows = O.groupby(cols, [0], aggs, 1 << 20)
    gt, grows = run(ctx, [cols], [0], aggs)
    assert_same(gt, grows, ot, orows, shape)


@pytest.mark.parametrize("slots,block,cap", [(64, 32, 0), (256, 96, 1024), (1024, 1024, 4096), (0, 64, 1024)])
@pytest.mark.parametrize("shape", ["head", "time"])
def test_private_tables_flush_and_grow(ctx, shape, slots, block, cap):
    # Small blocks take many windows per CTA (flushes that help and that do
    # not); a 1024-slot global table makes flushes and rows find no place.
    rng = np.random.default_rng(slots + block)
    cols = table(rng, keys_of(rng, shape, 200_003), True)
    cfg = qeg.agg_config(strategy=qeg.AGG_SMEM, smem_slots=slots, block_threads=block,
                         sizing=qeg.SIZE_FIXED if cap else qeg.SIZE_LEARNED, initial_capacity=cap)
    ot, orows = O.groupby(cols, [0], INT_F64, 1 << 20)
    gt, grows = run(ctx, [cols], [0], INT_F64, cfg)
    assert_same(gt, grows, ot, orows)


def test_private_tables_with_a_selection(ctx):
    rng = np.random.default_rng(3)
    cols = table(rng, keys_of(rng, "head", 50_000), True)
    sel = rng.integers(0, 50_000, 33_333).astype(np.uint32)  # repeats, any order
    sub = [O.TCol(c.type, c.values[sel], None if c.valid is None else c.valid[sel]) for c in cols]
    ot, orows = O.groupby(sub, [0], BARS, 1 << 20)
    gt, grows = run(ctx, [cols], [0], BARS, sel=sel)
    assert_same(gt, grows, ot, orows)


def small_column(rng, t, n, dictionary):
    if t == O.STR:
        return O.TCol(t, rng.integers(0, len(dictionary), n).astype(np.int32), None, dictionary)
    if t == O.BOOL:
        return O.TCol(t, rng.integers(0, 2, n).astype(np.uint8))
    return O.TCol(t, rng.integers(-3, 4, n).astype(np.int32))  # (0, 0) is key word 0


@pytest.mark.parametrize("ta", [O.I32, O.BOOL, O.STR])
@pytest.mark.parametrize("tb", [O.I32, O.BOOL, O.STR])
@pytest.mark.parametrize("nulls_from", [0, 1, 9])
def test_two_small_keys(ctx, ta, tb, nulls_from):
    """Three batches; from batch `nulls_from` on the second key has NULLs, so
    the packed table becomes composite rows there (0: it never packs)."""
    rng = np.random.default_rng(ta * 10 + tb)
    words = ["ab", "cd", "", "xyz"]
    canon = StrCanon(words)
    batches = []
    for b in range(3):
        n = 5_000 + 64 * b
        k2 = small_column(rng, tb, n, words)
        if b >= nulls_from:
            k2.valid = rng.random(n) >= 0.2
        batches.append([small_column(rng, ta, n, words[::-1]), k2, O.TCol(O.F64, rng.normal(0, 5, n), rng.random(n) > 0.1),
                        O.TCol(O.I32, rng.integers(-50, 50, n).astype(np.int32))])
    whole = [O.TCol(c.type, np.concatenate([b[i].values for b in batches]),
                    None if all(b[i].valid is None for b in batches) else
                    np.concatenate([np.ones(len(b[i].values), bool) if b[i].valid is None else b[i].valid for b in batches]),
                    c.dictionary) for i, c in enumerate(batches[0])]
    aggs = [(O.COUNT_STAR, 0), (O.SUM, 3), (O.AVG, 2), (O.MIN, 2), (O.MAX, 2)]
    ot, orows = O.groupby(whole, [0, 1], aggs, 1 << 20)
    gt, grows = run(ctx, batches, [0, 1], aggs, canon=canon)
    assert_same(gt, grows, ot, orows)


def test_two_i32_keys_large(ctx):
    # Above the sketch threshold, extreme values in both halves.
    rng = np.random.default_rng(8)
    n = 4_500_001
    a = rng.choice(np.array([-(1 << 31), -1, 0, 5, (1 << 31) - 1], np.int32), n)
    b = (rng.zipf(1.3, n) % 5_000 - 2_500).astype(np.int32)
    cols = [O.TCol(O.I32, a), O.TCol(O.I32, b), O.TCol(O.F64, rng.normal(0, 5, n), rng.random(n) > 0.05),
            O.TCol(O.I32, rng.integers(1, 100, n).astype(np.int32))]
    aggs = [(O.COUNT_STAR, 0), (O.SUM, 3), (O.AVG, 2), (O.MIN, 2), (O.MAX, 2), (O.COUNT, 2)]
    ot, orows = O.groupby(cols, [0, 1], aggs, 1 << 23)
    gt, grows = run(ctx, [cols], [0, 1], aggs)
    assert_same(gt, grows, ot, orows)


@pytest.mark.parametrize("aggs", [F64, BARS, WIDE, [(O.COUNT_STAR, 0), (O.MAX, 1)]],
                         ids=["f64", "bars", "wide", "generic_one"])
@pytest.mark.parametrize("bits", ["1", "7"])
def test_partitioned_passes_with_null_values(ctx, aggs, bits, monkeypatch):
    # Pool rows with validity bits; 2 partitions of 25,000 groups overflow their
    # tables and go to a 1M-slot global table, 128 do not.
    monkeypatch.setenv("QEG_AGG_PART_BITS", bits)
    rng = np.random.default_rng(int(bits))
    n = 150_001
    cols = table(rng, rng.integers(-(1 << 62), 1 << 62, n) // 7 % 50_000, True)
    ot, orows = O.groupby(cols, [0], aggs, 1 << 20)
    gt, grows = run(ctx, [cols], [0], aggs, qeg.agg_config(strategy=qeg.AGG_PARTITIONED))
    assert_same(gt, grows, ot, orows)


def test_two_i32_keys_partitioned(ctx):
    # Enough estimated groups for the partitioned passes, a heavy head, NULL
    # values; the groups come out of the tail rows.
    rng = np.random.default_rng(9)
    n = 4_400_003
    a = rng.integers(-4, 4, n).astype(np.int32)
    b = np.where(rng.random(n) < 0.5, rng.integers(0, 30, n), rng.integers(0, 150_000, n)).astype(np.int32)
    cols = [O.TCol(O.I32, a), O.TCol(O.I32, b), O.TCol(O.F64, rng.normal(0, 5, n), rng.random(n) > 0.05),
            O.TCol(O.I32, rng.integers(1, 100, n).astype(np.int32))]
    ot, orows = O.groupby(cols, [0, 1], [(O.SUM, 3), (O.AVG, 2)], 1 << 23)
    agg = qeg.Aggregate(ctx, [c.type for c in cols], [0, 1], [(O.SUM, 3), (O.AVG, 2)])
    agg.consume([to_gpu(c) for c in cols])
    agg.finish()
    assert agg.stats()["strategy"] == qeg.AGG_PARTITIONED, agg.stats()
    gt, grows = gpu_rows(agg.fetch(), agg.result_types)
    agg.close()
    assert_same(gt, grows, ot, orows)
