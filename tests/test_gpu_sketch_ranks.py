"""The sketch's ranking of heavy-hitter candidates when there are many of them
(sorts of 512 to 8192 estimates; the table of candidates holds that many), against numpy: the shares of the most
frequent keys, which stand clear of the rest."""
import numpy as np
import pytest
import torch

import qeg
from test_gpu_sketch_net import features, mix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [200, 400, 1000, 2500, 6000])
def test_many_candidates(tail):
    rng = np.random.default_rng(tail)
    hot = np.concatenate([rng.integers(3000, 5000, 128), rng.integers(300, 900, 128)])  # rows of each hot key
    keys = rng.permutation(1 << 20)[:256 + tail] * 0x1234567 + 1
    rows = np.repeat(keys[:256], hot)
    rows = rng.permutation(rows[:len(rows) // 4 * 4])
    # A tail key's four rows side by side: one CTA sees them, so it is a candidate.
    col = np.concatenate([rows, np.repeat(keys[256:], 4)]).reshape(-1, 4)
    col = np.ascontiguousarray(col[rng.permutation(len(col))].reshape(-1))
    assert len(col) < 1 << 20  # every row is sampled
    # The 128 largest count-min estimates are those of the 128 hottest keys.
    with np.errstate(over="ignore"):
        uniq, cnt = np.unique(col.astype(np.uint64), return_counts=True)
        h = mix64(uniq ^ np.uint64(0x243F6A8885A308D3))
        est = np.full(len(uniq), 1 << 60)
        for d in range(4):
            c = (mix64(h + np.uint64(0x9E3779B97F4A7C15 * (d + 1) & 0xFFFFFFFFFFFFFFFF)) >> np.uint64(40)).astype(np.int64) & 2047
            est = np.minimum(est, np.bincount(c, weights=cnt, minlength=2048)[c])
    top = np.argsort(est)[::-1][:128]
    assert set(uniq[top].tolist()) == set(keys[:128].tolist())
    ctx = qeg.Context(0)
    try:
        dev = torch.from_numpy(col).cuda()
        torch.cuda.synchronize()
        f, _, _ = qeg.sketch(ctx, qeg.Col(dev, None, qeg.I64))
    finally:
        ctx.close()
    exp = features(col.astype(np.uint64), 0)
    compared = [i for i in range(80) if i not in (72, 73)]  # (the 256 and 512 most frequent)
    assert np.allclose(f[compared], exp[compared], rtol=2e-7, atol=1e-9)
    assert f[71] <= f[72] <= f[73] <= 1.0
