"""GROUP BY over sequences of batches whose route changes on the way, against
the oracle: packed pairs of 4-byte keys that were partitioned and then meet a
NULL key, partitioned and preloaded private tables whose values gain NULLs,
packed tables that are nearly full, and a first batch that was refused."""
import numpy as np
import pytest

import oracle as O
import qeg
from util import assert_same, gpu_rows, to_gpu

pytestmark = pytest.mark.gpu


def whole(batches):
    """The batches as one table."""
    cols = []
    for i, c in enumerate(batches[0]):
        ok = None
        if any(b[i].valid is not None for b in batches):
            ok = np.concatenate([np.ones(b[i].n, bool) if b[i].valid is None else b[i].valid for b in batches])
        cols.append(O.TCol(c.type, np.concatenate([b[i].values for b in batches]), ok))
    return cols


def check(agg, batches, keys, aggs):
    agg.finish()
    gt, grows = gpu_rows(agg.fetch(), agg.result_types)
    ot, orows = O.groupby(whole(batches), keys, aggs, 1 << 23)
    assert_same(gt, grows, ot, orows)


@pytest.mark.parametrize("null_key", [0, 1])
def test_packed_pair_partitioned_then_null_keys(ctx, null_key):
    # The first batch's groups lie in the tail rows when the packing ends.
    rng = np.random.default_rng(11 + null_key)

    def batch(n, nulls):
        a = rng.integers(-4, 4, n).astype(np.int32)
        b = np.where(rng.random(n) < 0.5, rng.integers(0, 30, n), rng.integers(0, 150_000, n)).astype(np.int32)
        ok = rng.random(n) > 0.1 if nulls else None
        return [O.TCol(O.I32, a, ok if null_key == 0 else None), O.TCol(O.I32, b, ok if null_key == 1 else None),
                O.TCol(O.F64, rng.normal(0, 5, n)), O.TCol(O.I32, rng.integers(1, 100, n).astype(np.int32))]

    aggs = [(O.SUM, 3), (O.AVG, 2)]
    batches = [batch(4_400_003, False), batch(30_001, True), batch(20_000, False)]
    agg = qeg.Aggregate(ctx, [c.type for c in batches[0]], [0, 1], aggs)
    try:
        agg.consume([to_gpu(c) for c in batches[0]])
        assert agg.stats()["strategy"] == qeg.AGG_PARTITIONED, agg.stats()
        for b in batches[1:]:
            agg.consume([to_gpu(c) for c in b])
        check(agg, batches, [0, 1], aggs)
    finally:
        agg.close()


@pytest.mark.parametrize("strategy", [qeg.AGG_PARTITIONED, qeg.AGG_SMEM])
@pytest.mark.parametrize("ncols,t", [(2, O.F64), (3, O.I64)])
def test_values_gain_nulls(ctx, strategy, ncols, t):
    # As many private slots as fit without NULL counts: with them the same
    # number does not. The heavy hitters are preloaded.
    rng = np.random.default_rng(ncols)

    def batch(n, nulls):
        key = (30_000 ** rng.random(n)).astype(np.int64) - 1
        vals = [rng.normal(0, 9, n) if t == O.F64 else rng.integers(-99, 99, n) for _ in range(ncols)]
        return [O.TCol(O.I64, key * 0x51ED270B7)] + [O.TCol(t, v, rng.random(n) > 0.2 if nulls else None) for v in vals]

    batches = [batch(300_000, False), batch(200_003, True), batch(100_001, False)]
    aggs = [(f, c) for c in range(1, ncols + 1) for f in (O.SUM, O.MIN, O.MAX)]
    agg = qeg.Aggregate(ctx, [c.type for c in batches[0]], [0], aggs,
                        qeg.agg_config(strategy=strategy, hot_keys=4096, smem_slots=4096, expected_groups=30_000))
    try:
        for b in batches:
            agg.consume([to_gpu(c) for c in b])
            st = agg.stats()
            assert st["strategy"] == strategy and st["hot_keys"] > 500, st
        check(agg, batches, [0], aggs)
    finally:
        agg.close()


@pytest.mark.parametrize("seed", range(12))
def test_nearly_full_packed_table_meets_null_keys(ctx, seed):
    rng = np.random.default_rng(seed)
    cap = 1024 << (seed % 4)
    first = cap * 6 // 10 - 64  # (the table has first / 0.6 + 64 slots)
    keys = rng.permutation(1 << 24)[:cap * 82 // 100]  # 0.82 of its slots taken

    def batch(k, nulls):
        n = len(k)
        return [O.TCol(O.I32, (k >> 12).astype(np.int32)), O.TCol(O.I32, (k & 4095).astype(np.int32),
                rng.random(n) > 0.5 if nulls else None), O.TCol(O.I64, rng.integers(0, 9, n))]

    batches = [batch(keys[:first], False)] + [batch(p, False) for p in np.array_split(keys[first:], 8)]
    batches.append(batch(keys[:100], True))
    aggs = [(O.COUNT_STAR, 0), (O.SUM, 2)]
    agg = qeg.Aggregate(ctx, [c.type for c in batches[0]], [0, 1], aggs)
    try:
        for b in batches:
            agg.consume([to_gpu(c) for c in b])
        check(agg, batches, [0, 1], aggs)
    finally:
        agg.close()


def test_null_keys_after_a_refused_first_batch(ctx):
    # The first batch starts packed and is refused for its selection, before
    # there is a table; the next one has NULL keys.
    rng = np.random.default_rng(5)

    def batch(n, nulls):
        return [O.TCol(O.I32, rng.integers(0, 5, n).astype(np.int32)),
                O.TCol(O.I32, rng.integers(0, 5, n).astype(np.int32), rng.random(n) > 0.5 if nulls else None)]

    n = 4_300_000
    agg = qeg.Aggregate(ctx, [O.I32, O.I32], [0, 1], [(O.COUNT_STAR, 0)])
    try:
        with pytest.raises(qeg.QegError):
            agg.consume([to_gpu(c) for c in batch(n, False)], np.full(n, n, np.uint32))
        b = batch(10_000, True)
        agg.consume([to_gpu(c) for c in b])
        check(agg, [b], [0, 1], [(O.COUNT_STAR, 0)])
    finally:
        agg.close()
