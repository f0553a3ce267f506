"""Columns without NULLs read 32 bytes at a time: starts that are not aligned
to it, sizes around a vector, batches with and without NULLs mixed, and ranges
whose extreme value stands in the unaligned head or tail."""
import numpy as np
import pytest
import torch

import oracle as O
import qeg
from util import to_gpu

pytestmark = pytest.mark.gpu
NP = {O.I32: np.int32, O.I64: np.int64, O.TS: np.int64, O.F64: np.float64, O.BOOL: np.uint8}


def shifted(values, shift, type):
    """The values on the device, `shift` elements behind an aligned address."""
    t = torch.zeros(len(values) + shift, dtype=torch.from_numpy(values[:0]).dtype, device="cuda")
    t[shift:] = torch.from_numpy(values).cuda()
    torch.cuda.synchronize()
    return qeg.Col(t[shift:], None, type)


@pytest.mark.parametrize("sizes", [(1,), (3, 1), (31, 33, 4), (32, 32), (1000, 64, 7), (40001, 70000)])
@pytest.mark.parametrize("nulls", [None, 0, 1])  # the batch with NULLs (none of them; a size may not reach it)
@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("key", [O.I32, O.I64, O.BOOL])
def test_build_batches(ctx, sizes, nulls, shift, key):
    rng = np.random.default_rng(sum(sizes) + shift)
    n = sum(sizes)
    lim = 2 if key == O.BOOL else n
    kinds = [key, O.F64, O.I32, O.BOOL]
    vals = [(rng.permutation(n) % lim - (0 if key == O.BOOL else n // 2)).astype(NP[key]), rng.normal(0, 1, n),
            rng.integers(-9, 9, n).astype(np.int32), rng.integers(0, 2, n).astype(np.uint8)]
    valid = [np.ones(n, bool) for _ in kinds]
    j = qeg.Join(ctx, [key], kinds, [0], [0], qeg.LEFT)
    try:
        at, keep = 0, []
        for b, m in enumerate(sizes):
            cols = []
            for c, t in enumerate(kinds):
                v = np.ascontiguousarray(vals[c][at:at + m])
                if b == nulls and c != 2:
                    ok = rng.random(m) > 0.2
                    valid[c][at:at + m] = ok
                    cols.append(to_gpu(O.TCol(t, v, ok)))
                else:
                    cols.append(shifted(v, shift, t))
            keep.append(cols)
            j.build(cols)
            at += m
        j.build_finish()
        probe = np.unique(vals[0])
        if key == O.BOOL:
            probe = probe[:1]
        pcol = shifted(probe, shift, key)
        out_rows = j.probe([pcol])
        got = j.fetch(0, out_rows)
        exp = {}
        for r in range(n):
            if valid[0][r]:
                exp.setdefault(int(vals[0][r]), []).append(r)
        want = []
        for k in probe.tolist():
            for r in exp.get(k, [None]):
                want.append((k,) + ((None,) * 4 if r is None else tuple(
                    vals[c][r].item() if valid[c][r] else None for c in range(4))))
        rows = list(zip(*[[x if ok else None for x, ok in zip(v.tolist(), k.tolist())] for v, k in got]))
        order = lambda t: tuple((x is not None, x or 0) for x in t)
        assert sorted(rows, key=order) == sorted(want, key=order)
    finally:
        j.close()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 100, 70001])
@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("far", [0, -1, None])  # the time that does not fit a packed key
@pytest.mark.parametrize("time,key", [(O.TS, O.I32), (O.TS, O.I64), (O.I32, O.I64)])
def test_window_range(ctx, n, shift, far, time, key):
    rng = np.random.default_rng(n + shift)
    k = rng.integers(-5, 5, n).astype(NP[key])
    t = rng.integers(0, 1000, n).astype(NP[time])
    v = rng.integers(0, 100, n)
    if far is not None:
        if time == O.TS:
            t[far] = 1 << 40
        else:
            k[far] = -(1 << 40)
    w = qeg.Window(ctx, [key, time, O.I64], [0], 1, 10, [(qeg.COUNT_STAR, 0), (qeg.SUM, 2)])
    try:
        cols = [shifted(k, shift, key), shifted(t, shift, time), shifted(v, shift, O.I64)]
        w.consume(cols)
        w.finish()
        got = sorted(zip(*[x.tolist() for x, _ in w.fetch()]))
        b = t.astype(np.int64) // 10 * 10
        exp = {}
        for a, c, x in zip(k.tolist(), b.tolist(), v.tolist()):
            e = exp.setdefault((a, c), [0, 0])
            e[0] += 1
            e[1] += x
        assert [tuple(int(y) for y in g) for g in got] == sorted((a, c, e[0], e[1]) for (a, c), e in exp.items())
    finally:
        w.close()
