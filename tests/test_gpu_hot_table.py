"""The partitioned GROUP BY's table of heavy hitters (pairs of slots, keys moved
to their other pair when one is full): tables filled to the limit and beyond,
one key, the zero key among the heavy ones, values that reveal a row counted in
the wrong group."""
import numpy as np
import pytest

import oracle as O
import qeg
from util import to_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [64, 256, 4096])
@pytest.mark.parametrize("hot", [1, 2, 16, 55, 218, 3481, 4096])
@pytest.mark.parametrize("nulls", [False, True])
def test_hot_table(ctx, slots, hot, nulls):
    rng = np.random.default_rng(slots + hot)
    n, dom = 400000, 30000
    r = np.minimum((dom ** rng.random(n)).astype(np.int64) - 1, dom - 1)
    key = r * 0x51ED270B7F4A7C15 % (1 << 62)  # the most frequent one is 0
    ok = rng.random(n) > 0.02 if nulls else np.ones(n, bool)
    val = key % 1009 + rng.integers(0, 3, n)
    a = qeg.Aggregate(ctx, [qeg.I64, qeg.I64], [0], [(qeg.COUNT_STAR, 0), (qeg.SUM, 1), (qeg.MIN, 1), (qeg.MAX, 1)],
                      qeg.agg_config(strategy=qeg.AGG_PARTITIONED, hot_keys=hot, smem_slots=slots,
                                     expected_groups=dom))
    try:
        a.consume([to_gpu(O.TCol(O.I64, key, ok if nulls else None)), to_gpu(O.TCol(O.I64, val))])
        groups = a.finish()
        st = a.stats()
        assert st["strategy"] == qeg.AGG_PARTITIONED and 0 < st["hot_keys"] <= min(hot, slots * 17 // 20)
        # All asked for are found a place while the table is half empty.
        assert hot > slots // 2 or st["hot_keys"] == hot
        got = {}
        for row in zip(*[[x if v else None for x, v in zip(vals.tolist(), valid.tolist())] for vals, valid in a.fetch()]):
            got[row[0]] = row[1:]
    finally:
        a.close()
    k = np.where(ok, key, -1)
    uniq, inv = np.unique(k, return_inverse=True)
    cnt, total = np.bincount(inv), np.zeros(len(uniq), np.int64)
    lo, hi = np.full(len(uniq), 1 << 60), np.full(len(uniq), -1)
    np.add.at(total, inv, val)
    np.minimum.at(lo, inv, val)
    np.maximum.at(hi, inv, val)
    assert groups == len(uniq) == len(got)
    for i, u in enumerate(uniq.tolist()):
        assert got[None if u == -1 else u] == (cnt[i], total[i], lo[i], hi[i])
