"""The fused pipeline's typed kernel at the row count where one launch ends and
the next begins (its per-lane 32-bit counts and sum halves are full there):
every row in one group, quantities whose halves are at their extremes."""
import pytest

import qeg

pytestmark = pytest.mark.gpu


def test_rows_beyond_one_launch(ctx):
    torch = pytest.importorskip("torch")
    # One launch takes 32 * 65,024 rows per CTA, of which an SM holds one or two.
    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count * 32 * 65024 + 12_345
    key = torch.zeros(n, dtype=torch.int32, device="cuda")
    price = torch.ones(n, dtype=torch.float64, device="cuda")
    bkey, sector = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (0, 9))
    try:
        for q in (65535, -1, -(1 << 31), (1 << 31) - 1):
            qty = torch.full((n,), q, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            for rows in (n, n // 2 + 1):  # two launches, or the end of one
                _, res = qeg.filter_join_agg(ctx, [qeg.Col(c[:rows]) for c in (key, price, qty)],
                                             [qeg.Col(bkey), qeg.Col(sector)], 0, 0, 4,
                                             [(qeg.COUNT_STAR, 0), (qeg.AVG, 1), (qeg.SUM, 2)], filter_col=1,
                                             filter_op=qeg.CMP_GT, filter_value=0.5)
                assert [v.tolist() for v, _ in res] == [[9], [rows], [1.0], [q * rows]], (q, rows)
            del qty
    finally:
        del key, price
        torch.cuda.empty_cache()
