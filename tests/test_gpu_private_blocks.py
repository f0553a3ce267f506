"""CTA-private GROUP BY tables in blocks of fewer than 1024 threads, several of
which share an SM, against the oracle: tables that overflow into a global
table that has to grow, so rows of every block's last flush are left over."""
import numpy as np
import pytest

import oracle as O
import qeg
from test_gpu_private import INT_F64, keys_of, run, table
from util import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,block", [(64, 32), (64, 128), (1024, 256), (0, 256), (2048, 512)])
@pytest.mark.parametrize("nulls", [False, True])
def test_blocks_that_share_an_sm(ctx, slots, block, nulls):
    rng = np.random.default_rng(slots + block)
    cols = table(rng, keys_of(rng, "many", 2_600_003), nulls)
    cfg = qeg.agg_config(strategy=qeg.AGG_SMEM, smem_slots=slots, block_threads=block, sizing=qeg.SIZE_FIXED,
                         initial_capacity=4096)
    gt, grows = run(ctx, [cols, [O.TCol(c.type, c.values[:999], None if c.valid is None else c.valid[:999]) for c in cols]],
                    [0], INT_F64, cfg)
    both = [O.TCol(c.type, np.concatenate([c.values, c.values[:999]]),
                   None if c.valid is None else np.concatenate([c.valid, c.valid[:999]])) for c in cols]
    ot, orows = O.groupby(both, [0], INT_F64, 1 << 22)
    assert_same(gt, grows, ot, orows)
