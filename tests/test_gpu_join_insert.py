"""Inserts of a hashed single-key build side, a bucket per step: sizes around a
thread's rows and a grid's step, keys repeated by neighbouring threads (claims
lost to the same and to other keys), the zero key, NULL keys, with and without
the Bloom filter."""
import numpy as np
import pytest

import oracle as O
import qeg
from util import to_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bloom", ["0", "1"])
@pytest.mark.parametrize("n", [1, 2, 255, 257, 600001, 1300007])
@pytest.mark.parametrize("repeat", [1, 2, 64, 5000])
def test_insert(ctx, monkeypatch, n, repeat, bloom):
    monkeypatch.setenv("QEG_JOIN_BLOOM", bloom)
    rng = np.random.default_rng(n + repeat)
    ids = np.arange(n) // repeat  # repeats side by side: the same warp claims one slot
    if repeat == 2:
        ids = rng.permutation(ids)
    keys = ids * 0x51ED270B7F4A7C15 % (1 << 62)  # 0 is among them
    ok = rng.random(n) > 0.05 if n > 2 else np.ones(n, bool)
    probe = np.concatenate([np.unique(keys), np.arange(1, 1000) * 3 + (1 << 61)])
    val = rng.integers(-1000, 1000, len(probe))
    j = qeg.Join(ctx, [qeg.I64, qeg.I64], [qeg.I64], [0], [0], qeg.INNER)
    try:
        bcol = to_gpu(O.TCol(O.I64, keys, None if ok.all() else ok))
        pk, pv = to_gpu(O.TCol(O.I64, probe)), to_gpu(O.TCol(O.I64, val))
        j.build([bcol])
        j.build_finish()
        uniq, cnt = np.unique(keys[ok], return_counts=True)
        assert j.stats()["distinct_keys"] == len(uniq)
        at = np.minimum(np.searchsorted(uniq, probe), max(len(uniq) - 1, 0))
        mult = np.where(uniq[at] == probe, cnt[at], 0) if len(uniq) else np.zeros(len(probe), np.int64)
        j.probe_count_sum(pk, pv)
        count, total = j.count_sum()
        assert count == mult.sum()
        assert (total or 0) == (mult * val).sum()
    finally:
        j.close()
