"""Estimate-sized join tables give up an insert after 1024 slots: build keys
that share a home bucket, fewer and more of them than that, against numpy."""
import numpy as np
import pytest

import qeg

pytestmark = pytest.mark.gpu

M = (1 << 64) - 1
A, B = 0x9E3779B97F4A7C15, 0xD1342543DE82EF95


def key_of_hash(h):
    """The key whose hash (two multiplies, a bijection) is h."""
    x = h * pow(B, -1, 1 << 64) & M
    return (x ^ (x >> 32)) * pow(A, -1, 1 << 64) & M


@pytest.mark.parametrize("cluster,rebuilds", [(600, 0), (1600, 1)])
def test_full_neighbourhood(ctx, cluster, rebuilds):
    rng = np.random.default_rng(cluster)
    # 96k other keys; 4 slots per estimated key make 2^19 slots, and the top 19
    # bits of these hashes are the same.
    same = [key_of_hash((0x2A5A8 << 45) | int(x)) for x in np.unique(rng.integers(0, 1 << 45, cluster))]
    keys = np.unique(np.concatenate([np.array(same, np.uint64).view(np.int64), rng.integers(1 << 40, 1 << 62, 96_000)]))
    build = rng.permutation(np.repeat(keys, 11))
    probe = np.concatenate([keys, keys + 1])
    val = rng.integers(-1000, 1000, len(probe))
    j = qeg.Join(ctx, [qeg.I64, qeg.I64], [qeg.I64], [0], [0], qeg.INNER, strategy=qeg.JOIN_HASH)
    try:
        j.build([qeg.Col(build)])
        j.build_finish()
        st = j.stats()
        assert st["slots"] > 1 << 19 if rebuilds else st["slots"] == 1 << 19, st
        assert st["rebuilds"] == rebuilds, st
        j.probe_count_sum(qeg.Col(probe), qeg.Col(val))
        mult = 11 * np.isin(probe, keys)
        assert j.count_sum() == (mult.sum(), (mult * val).sum())
    finally:
        j.close()
