"""The fused pipeline's typed trades kernel against numpy: 32-bit quantities at
their extremes (their 64-bit sums are kept in 16-bit halves), prices around a
positive literal that differ in their low or high 32 bits only, subnormal and
huge literals, and row counts around the kernel's tiles."""
import numpy as np
import pytest

import qeg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 5120, 100_003])
@pytest.mark.parametrize("lit", [100.0, 5e-324, 1e308, -1.5])
@pytest.mark.parametrize("op", [qeg.CMP_LT, qeg.CMP_LE, qeg.CMP_GT, qeg.CMP_GE, qeg.CMP_EQ, qeg.CMP_NE])
def test_quantity_halves_and_literal_halves(ctx, n, lit, op):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + op)
    nsym, sectors = 50, 7
    sector = rng.integers(0, sectors, nsym).astype(np.int32)
    sym = rng.integers(-2, nsym + 2, n).astype(np.int32)  # some keys outside the table
    near = [lit, np.nextafter(lit, 1e9), np.nextafter(lit, -1e9), -lit, lit * 2, 0.0, -0.0]
    price = rng.choice(np.array(near), n)
    qty = rng.choice(np.array([-(1 << 31), (1 << 31) - 1, -1, 0, 1, 65535, 65536, -65536, -65537], np.int32), n)
    dev = [torch.from_numpy(x).cuda() for x in (sym, price, qty, np.arange(nsym, dtype=np.int32), sector)]
    torch.cuda.synchronize()
    _, res = qeg.filter_join_agg(ctx, [qeg.Col(d) for d in dev[:3]], [qeg.Col(d) for d in dev[3:]], 0, 0, 4,
                                 [(qeg.COUNT_STAR, 0), (qeg.AVG, 1), (qeg.SUM, 2)], filter_col=1, filter_op=op,
                                 filter_value=lit)
    f = {qeg.CMP_LT: np.less, qeg.CMP_LE: np.less_equal, qeg.CMP_GT: np.greater, qeg.CMP_GE: np.greater_equal,
         qeg.CMP_EQ: np.equal, qeg.CMP_NE: np.not_equal}[op]
    keep = f(price, lit) & (sym >= 0) & (sym < nsym)
    got = {int(k): (int(c), float(a), int(s)) for k, c, a, s in zip(*[v for v, _ in res])}
    want = {}
    for g in range(sectors):
        rows = keep & (sector[np.clip(sym, 0, nsym - 1)] == g)
        if rows.any():
            want[g] = (int(rows.sum()), price[rows], int(qty[rows].astype(np.int64).sum()))
    assert got.keys() == want.keys()
    for g, (c, p, s) in want.items():
        assert got[g][0] == c and got[g][2] == s
        # Sums of at most c terms in any order: c * eps * sum of magnitudes, per row.
        with np.errstate(over="ignore"):
            bound = c * 2.0 ** -52 * float(np.abs(p / c).sum())
            total, finite = float(p.sum()), bool(np.isfinite(np.abs(p).sum()))
        assert not finite or abs(got[g][1] - total / c) <= bound
