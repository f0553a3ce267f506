"""The sketch of a key column and the estimate drawn from it in the same
launch, against numpy: registers, count-min ranks of the most frequent keys
(sort sizes below, at and above a warp's and a padded power of two), NULLs, and
the network's outputs for those features."""
import numpy as np
import pytest
import torch

import qeg

pytestmark = pytest.mark.gpu


def mix64(x):
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def features(words, nulls):
    """The 80 features of a fully sampled column, in float64."""
    with np.errstate(over="ignore"):
        h = mix64(words ^ np.uint64(0x243F6A8885A308D3))
        regs = np.zeros(1 << 14, np.int64)
        rest = (h << np.uint64(14)) | np.uint64(1 << 13)
        rho = 64 - np.floor(np.log2(rest.astype(np.float64) / 2.0 ** 64) + 64).astype(np.int64)
        np.maximum.at(regs, (h >> np.uint64(50)).astype(np.int64), rho)
        keys, cnt = np.unique(words, return_counts=True)
        hk = mix64(keys ^ np.uint64(0x243F6A8885A308D3))
        est = np.full(len(keys), 1 << 60)
        for d in range(4):
            c = (mix64(hk + np.uint64(0x9E3779B97F4A7C15 * (d + 1) & 0xFFFFFFFFFFFFFFFF)) >> np.uint64(40)).astype(np.int64) & 2047
            row = np.bincount(c, weights=cnt, minlength=2048)
            est = np.minimum(est, row[c])
            if d == 0:
                f2 = float((row ** 2).sum())
    f = np.zeros(80)
    np.add.at(f, np.minimum(regs, 63), 1.0 / (1 << 14))
    ranked = np.sort(est)[::-1]
    n = len(words)
    for i in range(10):
        f[64 + i] = min(1.0, ranked[:1 << i].sum() / n)
    f[74] = f2 / n ** 2
    f[75] = f[76] = np.log2(1.0 + n + nulls) / 32
    f[77] = 1.0
    f[78] = nulls / (n + nulls)
    m = float(1 << 14)
    e = (0.7213 / (1 + 1.079 / m)) * m * m / (2.0 ** -regs.astype(np.float64)).sum()
    zeros = (regs == 0).sum()
    if e <= 2.5 * m and zeros:
        e = m * np.log(m / zeros)
    f[79] = min(1.0, e / n)
    return f


@pytest.mark.parametrize("distinct", [1, 2, 31, 33, 255, 256, 257, 300])
@pytest.mark.parametrize("rows,null_pct", [(70001, 0), (262144, 10)])
def test_sketch_and_network(distinct, rows, null_pct):
    ctx = qeg.Context(0)
    try:
        rng = np.random.default_rng(distinct + rows)
        key = rng.integers(1, distinct + 1, rows) * 0x1234567
        ok = rng.random(rows) >= null_pct / 100
        bits = np.packbits(np.concatenate([ok, np.zeros(-rows % 64, bool)]), bitorder="little").view(np.int64)
        col = qeg.Col(torch.from_numpy(key).cuda(), torch.from_numpy(bits).cuda() if null_pct else None, qeg.I64)
        f, classic, top = qeg.sketch(ctx, col)
        exp = features(key[ok if null_pct else slice(None)].astype(np.uint64), int((~ok).sum()) if null_pct else 0)
        # Features are float32 of values in [0, 1]; the sums behind them are exact.
        assert np.allclose(f, exp, rtol=2e-7, atol=1e-9)
        if distinct <= 256:
            assert abs(top - 1.0) < 1e-12
    finally:
        ctx.close()


@pytest.mark.parametrize("distinct", [1, 33, 256, 300])
def test_estimate_uses_the_network(distinct):
    """The group estimate of a GROUP BY is the network's for the sketch's
    features (computed apart here); a sample of a quarter of the rows."""
    ctx = qeg.Context(0)
    try:
        rows = 1 << 22
        key = torch.randint(1, distinct + 1, (rows,), device="cuda", dtype=torch.int64) * 0x1234567
        torch.cuda.synchronize()
        col = qeg.Col(key, None, qeg.I64)
        f, classic, _ = qeg.sketch(ctx, col)
        a = qeg.Aggregate(ctx, [qeg.I64], [0], [(qeg.COUNT_STAR, 0)], qeg.agg_config(sizing=qeg.SIZE_LEARNED))
        a.consume([col])
        a.finish()
        est = a.stats()["est_groups"]
        a.close()
        g = qeg.learned_groups(classic, float(qeg.estimator_predict(ctx, f)[0][0]), qeg.estimator_get_deadband(ctx))
        # Bounded below by 0.95 times the sample's distinct count.
        sample = float(f[79]) * round(2.0 ** (float(f[75]) * 32) - 1)
        g = max(g, 0.95 * sample, 1.0)
        assert abs(est - g) <= 1e-4 * g, (est, g)
    finally:
        ctx.close()
