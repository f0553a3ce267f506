"""The fused pipeline over STR keys whose build side repeats a key: one that no
probe key refers to, one that some do, none, against numpy and with every
kernel's choice of group lists."""
import numpy as np
import pytest

import qeg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [None, "shared"])
@pytest.mark.parametrize("repeated", ["none", "unseen", "seen"])
@pytest.mark.parametrize("nsym", [3, 40, 3000])
def test_repeated_build_keys(ctx, kernel, repeated, nsym, monkeypatch):
    torch = pytest.importorskip("torch")
    if kernel:
        monkeypatch.setenv("QEG_PIPE_KERNEL", kernel)
    rng = np.random.default_rng(nsym)
    n, sectors = 70_001, 6
    code = rng.integers(0, nsym, n).astype(np.int32)
    price, qty = rng.uniform(0, 100, n), rng.integers(-50, 50, n).astype(np.int32)
    # Build dictionary: the probe's strings in another order, and one more.
    perm = rng.permutation(nsym + 1).astype(np.int32)  # build code -> value id (nsym: not in the probe's dictionary)
    bcode = np.arange(nsym + 1, dtype=np.int32)
    again = {"none": [], "unseen": [int(np.flatnonzero(perm == nsym)[0])], "seen": [int(np.flatnonzero(perm == 1)[0])]}
    bcode = np.concatenate([bcode, np.array(again[repeated], np.int32)])
    sector = rng.integers(0, sectors, len(bcode)).astype(np.int32)
    dev = [torch.from_numpy(x).cuda() for x in (code, price, qty, bcode, sector, np.arange(nsym, dtype=np.int32), perm)]
    torch.cuda.synchronize()
    _, res = qeg.filter_join_agg(ctx, [qeg.Col(dev[0], None, qeg.STR, dev[5]), qeg.Col(dev[1]), qeg.Col(dev[2])],
                                 [qeg.Col(dev[3], None, qeg.STR, dev[6]), qeg.Col(dev[4])], 0, 0, 4,
                                 [(qeg.COUNT_STAR, 0), (qeg.AVG, 1), (qeg.SUM, 2)], filter_col=1,
                                 filter_op=qeg.CMP_GT, filter_value=25.0)
    keep = price > 25.0
    want = np.zeros((sectors, 3))
    for b, g in zip(bcode, sector):
        rows = keep & (code == perm[b]) if perm[b] < nsym else np.zeros(n, bool)
        want[g] += [rows.sum(), price[rows].sum(), qty[rows].astype(np.int64).sum()]
    got = {int(k): (int(c), float(a), int(s)) for k, c, a, s in zip(*[v for v, _ in res])}
    assert got.keys() == {g for g in range(sectors) if want[g][0]}
    for g, (c, a, s) in got.items():
        assert (c, s) == (want[g][0], want[g][2])
        assert abs(a - want[g][1] / c) <= 2 * c * 2.0 ** -52 * 100.0  # two sums of c terms below 100, in any order
