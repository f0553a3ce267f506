"""Calls that take memory for speed alone answer without it: joins whose build
rows cannot be packed side by side, partitioned GROUP BYs without their pool, as-of joins without the
merge's scratch."""
import numpy as np
import pytest
import torch

import oracle as O
import qeg
from mempool import limited_pool
from test_gpu_asof_merge import expected
from util import to_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("join_type", [O.INNER, O.LEFT])
def test_fetch_without_room_for_packed_rows(ctx, device, join_type):
    rng = np.random.default_rng(2)
    nb, n = 1 << 22, 2_400_000  # packed: 64 bytes a row, 256 MB
    bkey = rng.permutation(nb) * 0x51ED270B7
    build = [O.TCol(O.I64, bkey)] + [O.TCol(O.I64, rng.integers(0, 1 << 40, nb), rng.random(nb) > 0.1 if c else None)
                                     for c in range(4)]
    at = rng.integers(0, nb, n)
    miss = rng.random(n) < 0.1
    probe = [O.TCol(O.I64, np.where(miss, -1, bkey[at])), O.TCol(O.I32, np.arange(n, dtype=np.int32), rng.random(n) > 0.3)]
    j = qeg.Join(ctx, [c.type for c in probe], [c.type for c in build], [0], [0], join_type)
    try:
        j.build([to_gpu(c, device=True) for c in build])
        j.build_finish()
        cols = [to_gpu(c, device=True) for c in probe]
        m = j.probe(cols)
        keep = np.arange(n) if join_type == O.LEFT else np.flatnonzero(~miss)
        assert m == len(keep)
        with limited_pool(224 << 20):
            got = j.fetch_device() if device else j.fetch()
            ctx.synchronize()
        with pytest.raises(qeg.QegError):  # (the pool is as small as it says)
            with limited_pool(32 << 20):
                k = qeg.Join(ctx, [O.I64], [O.I64] * 5, [0], [0], O.INNER)
                try:
                    k.build([to_gpu(c, device=True) for c in build])
                finally:
                    k.close()
                    ctx.synchronize()
        for c, (v, w) in enumerate(got):
            if device:
                v, w = v[:m].cpu().numpy(), qeg.unpack_validity(w.cpu().numpy().view(np.uint64), m)
            src = probe[c] if c < 2 else build[c - 2]
            row = keep if c < 2 else at[keep]
            ok = np.ones(len(src.values), bool) if src.valid is None else src.valid
            ok = ok[row] if c < 2 else ok[row] & ~miss[keep]
            assert np.array_equal(w, ok), c
            assert np.array_equal(v[ok], src.values[row][ok]), c
    finally:
        j.close()
        torch.cuda.synchronize()


@pytest.mark.parametrize("hot_keys", [0, 64])
@pytest.mark.parametrize("expected,mb", [(100_000, 112), (12_000_000, 288)])
def test_partitioned_groupby_without_room_for_its_pool(ctx, hot_keys, expected, mb):
    # The pool would take 16 bytes a row, up to 128 MB; the rest fits. Or the
    # pool fits and the tail rows, 16 bytes for 1.25 of the expected groups, do
    # not (240 MB).
    n, dom = 1 << 23, 100_000
    g = torch.Generator(device="cuda").manual_seed(4)
    a = qeg.Aggregate(ctx, [O.I64], [0], [(O.COUNT_STAR, 0)],
                      qeg.agg_config(strategy=qeg.AGG_PARTITIONED, hot_keys=hot_keys, expected_groups=expected))
    try:
        want = torch.zeros(dom, dtype=torch.int64, device="cuda")
        for limit in (mb << 20, mb << 20, 0):  # twice without that memory, then with it
            key = (dom ** torch.rand(n, device="cuda", dtype=torch.float64, generator=g)).long() - 1
            want += torch.bincount(key, minlength=dom)
            torch.cuda.synchronize()
            if limit:
                with limited_pool(limit):
                    a.consume([qeg.Col(key)])
                    ctx.synchronize()
            else:
                a.consume([qeg.Col(key)])
        assert a.finish() == int((want > 0).sum())
        (k, _), (c, _) = a.fetch()
        assert a.stats()["strategy"] == qeg.AGG_PARTITIONED
        got = np.zeros(dom, np.int64)
        got[k] = c
        assert np.array_equal(got, want.cpu().numpy())
    finally:
        a.close()


def test_asof_without_room_for_the_merge(ctx):
    # 16,000 slots and as many slices as fill the GPU take about 30 MB; the probe
    # batch's own buffers 8 MB. The build side was sorted by an earlier batch.
    rng = np.random.default_rng(6)
    nb, n, nsym = 100_000, 2_000_000, 16_000
    bts, pts = np.sort(rng.integers(0, 1 << 30, nb)), np.sort(rng.integers(0, 1 << 30, n))
    bkey, pkey = rng.integers(0, nsym, nb).astype(np.int32), rng.integers(0, nsym, n).astype(np.int32)
    exp = expected(bkey.astype(np.int64), bts, pkey.astype(np.int64), pts, None)
    j = qeg.AsofJoin(ctx, [O.I32, O.TS], [O.I32, O.TS, O.I64], [0], [0], 1, 1, O.LEFT)
    try:
        j.build([qeg.Col(bkey), qeg.Col(bts, None, qeg.TS), qeg.Col(np.arange(nb))])
        j.build_finish()
        assert j.probe([qeg.Col(pkey[:50_000]), qeg.Col(pts[:50_000], None, qeg.TS)]) == 50_000  # (fewer rows: the search)
        cols = [to_gpu(O.TCol(O.I32, pkey), device=True), to_gpu(O.TCol(O.TS, pts), device=True)]
        with limited_pool(32 << 20):
            assert j.probe(cols) == n
            ctx.synchronize()
        v, ok = j.fetch()[-1]
        assert np.array_equal(np.where(ok, v, -1), exp)
        assert j.probe(cols) == n  # with memory again
        v, ok = j.fetch()[-1]
        assert np.array_equal(np.where(ok, v, -1), exp)
    finally:
        j.close()
