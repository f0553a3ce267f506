"""As-of join of a build side in time order with probe rows that are not, but
whose disorder is rare: sorted runs one behind the other, so that hardly any
neighbouring pair is out of order and the ends of the merge's slices step back.
The answer has to be the search's."""
import numpy as np
import pytest

import oracle as O
import qeg
from test_gpu_asof_merge import expected, run

pytestmark = pytest.mark.gpu


def order_of(rng, shape, n, key):
    """A permutation of n rows in time order."""
    if shape == "two_runs":  # every other row, then the rest
        return np.concatenate([np.arange(0, n, 2), np.arange(1, n, 2)])
    if shape == "seven_runs":
        return np.concatenate([np.arange(i, n, 7) for i in range(7)])
    if shape == "rotated":  # the last third first
        return np.roll(np.arange(n), n // 3)
    if shape == "late_block":  # one block of early rows at the end
        return np.concatenate([np.arange(1000), np.arange(1400, n), np.arange(1000, 1400)])
    if shape == "by_key":
        return np.argsort(key, kind="stable")
    return np.arange(n)[::-1]


@pytest.mark.parametrize("shape", ["two_runs", "seven_runs", "rotated", "late_block", "by_key", "backwards"])
@pytest.mark.parametrize("nb,npr,nsym", [(3000, 3500, 20), (200_000, 400_000, 500), (300_001, 300_007, 3)])
@pytest.mark.parametrize("plain", [True, False])
def test_probe_of_sorted_runs(ctx, shape, nb, npr, nsym, plain):
    rng = np.random.default_rng(nb + nsym)
    bts, pts = np.sort(rng.integers(0, 1 << 30, nb)), np.sort(rng.integers(0, 1 << 30, npr))
    bkey, pkey = rng.integers(0, nsym, nb), rng.integers(0, nsym, npr)
    perm = order_of(rng, shape, npr, pkey)
    pts, pkey = pts[perm], pkey[perm]
    exp = expected(bkey, bts, pkey, pts, None)

    def side(k, t, n):
        key = O.TCol(O.I32, k.astype(np.int32)) if plain else O.TCol(O.I64, k * 0x51ED270B7 + 3)
        return [key, O.TCol(O.TS, t), O.TCol(O.I64, np.arange(n))]

    build, probe = side(bkey, bts, nb), side(pkey, pts, npr)
    assert np.array_equal(run(ctx, build, probe, 1, O.LEFT, None), exp)
    # A batch in time order, then one that is not (the merge, then the search).
    first = np.argsort(pts[:npr // 2], kind="stable")
    perm = np.concatenate([first, np.arange(npr // 2, npr)])
    both = [O.TCol(c.type, c.values[perm]) for c in probe]
    assert np.array_equal(run(ctx, build, both, 1, O.INNER, None, 2), exp[perm][exp[perm] >= 0])
