"""Materialised joins with repeated build keys whose table slots are carried as
64-bit numbers (as for tables of 2^32-1 slots or more), against the oracle."""
import numpy as np
import pytest

import oracle as O
import qeg
from test_gpu_join_rows import build_keys, check, columns
from util import to_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_rows", [1, 65, 4097])
@pytest.mark.parametrize("join_type", [O.INNER, O.LEFT])
@pytest.mark.parametrize("kind,nkeys", [("dense", 1), ("sparse", 1), ("sparse", 3)])
def test_wide_slots(ctx, np_rows, join_type, kind, nkeys, monkeypatch):
    monkeypatch.setenv("QEG_JOIN_WIDE_SLOTS", "1")
    rng = np.random.default_rng(np_rows + nkeys)
    nb = 900
    bids = build_keys(rng, nb, kind, 3)
    pids = np.where(rng.random(np_rows) < 0.6, bids[rng.integers(0, nb, np_rows)], -5 - np.arange(np_rows))
    build = columns(rng, nb, nkeys, bids, 3) + [O.TCol(O.I64, np.arange(nb))]
    probe = columns(rng, np_rows, nkeys, pids, 3) + [O.TCol(O.I64, np.arange(np_rows))]
    on = list(range(nkeys))
    et, erows = O.join(probe, build, on, on, join_type)
    j = qeg.Join(ctx, [c.type for c in probe], [c.type for c in build], on, on, join_type)
    try:
        j.build([to_gpu(c) for c in build])
        j.build_finish()
        j.probe([to_gpu(c) for c in probe])
        check(et, j.fetch(), erows)
    finally:
        j.close()
