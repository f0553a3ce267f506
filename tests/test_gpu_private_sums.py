"""Single-key GROUP BY through private tables that keep F64 sums in shared
memory (chosen when the expected groups make a global table beyond L2), against
the oracle: every field set, rows of a warp on one slot (replicas), tables that
are flushed and refilled, infinities and NaN, few rows and small blocks."""
import numpy as np
import pytest

import oracle as O
import qeg
from test_gpu_private import BARS, F64, INT_F64, WIDE, keys_of, run, table
from util import assert_same

pytestmark = pytest.mark.gpu

SUMS4 = [(O.SUM, 2), (O.AVG, 4), (O.SUM, 5), (O.SUM, 6), (O.COUNT, 2)]


@pytest.mark.parametrize("shape", ["one", "few", "head", "many", "time"])
@pytest.mark.parametrize("aggs,nulls", [(INT_F64, False), (INT_F64, True), (F64, False), (F64, True), (BARS, False),
                                        (BARS, True), (WIDE, True), (SUMS4, True), ([(O.SUM, 2)], True)],
                         ids=["int_f64", "int_f64_nulls", "f64", "f64_nulls", "bars", "bars_nulls", "wide", "sums4", "sum"])
def test_shared_sums(ctx, shape, aggs, nulls):
    rng = np.random.default_rng(len(shape) * 100 + len(aggs) * 2 + nulls)
    n = 300_007
    cols = table(rng, keys_of(rng, shape, n), nulls)
    cols += [O.TCol(O.F64, rng.normal(0, 1e3, n), rng.random(n) > 0.2 if nulls else None) for _ in range(3)]
    ot, orows = O.groupby(cols, [0], aggs, 1 << 20)
    gt, grows = run(ctx, [cols], [0], aggs, qeg.agg_config(strategy=qeg.AGG_SMEM, expected_groups=20_000_000))
    assert_same(gt, grows, ot, orows, shape)


@pytest.mark.parametrize("slots,block", [(64, 32), (256, 256), (0, 96)])
@pytest.mark.parametrize("n", [1, 4097, 900_001])
def test_shared_sums_small_blocks_and_extremes(ctx, slots, block, n):
    rng = np.random.default_rng(slots + n)
    cols = table(rng, keys_of(rng, "head", n), True)
    v = cols[2].values
    v[rng.random(n) < 0.001] = np.inf  # its group's sum is inf, or NaN with the next line's rows
    v[rng.random(n) < 0.0005] = -np.inf
    v[rng.random(n) < 0.0005] = np.nan
    v[rng.random(n) < 0.01] = -0.0
    cfg = qeg.agg_config(strategy=qeg.AGG_SMEM, expected_groups=20_000_000, smem_slots=slots, block_threads=block)
    ot, orows = O.groupby(cols, [0], F64, 1 << 21)
    gt, grows = run(ctx, [cols], [0], F64, cfg)
    assert_same(gt, grows, ot, orows)
