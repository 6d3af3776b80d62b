"""group_id where its dispatch turns (k_group.cu): the numbering by ranks and by lookback, the table that
must hold every key, the first table and its giving up, and the regions' steps; few, many and skewed
keys. And bucket sums and counts over groups of 32 rows with and without equal neighbours (k_index.cu)."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def keys(kind, n, seed):
    u = oracle.rand_i64(n, seed).view(np.uint64)
    if kind == "all":
        return u.view(np.int64)
    if kind == "skewed":
        return (np.uint64(1) << (u % np.uint64(64))).view(np.int64)
    if kind == "late":  # a key that only the last rows hold
        k = (u % np.uint64(7)).astype(np.int64)
        k[-3:] = -2**63
        return k
    return (u % np.uint64(kind)).astype(np.int64) * 0x1E3779B97F4A7C15


@pytest.mark.parametrize("n", [4095, 70_001, (1 << 20) + 1, (1 << 22) - 1, (1 << 22) + 33])
def test_group_ids(ctx, n):
    for kind in (10, 4096, 300_000, 3_000_000, "all", "skewed", "late"):
        k = keys(kind, n, n)
        assert np.array_equal(ctx.call("group_id_i64", ctx.upload(k)).numpy(), oracle.group_id_i64(k)), kind
    a, b = keys(1000, n, 1), keys(700, n, 2)
    got = ctx.call("group_id2_i64_i64", ctx.upload(a), ctx.upload(b)).numpy()
    assert np.array_equal(got, oracle.group_id2_i64_i64(a, b))


def test_bucket_groups(ctx):
    n = 100_003
    u = oracle.rand_i64(n, 4).view(np.uint64)
    v = oracle.rand_i64(n, 5)
    v[::3] = -1  # carries into the high words
    alternating = np.arange(n, dtype=np.int64) % 2
    low_equal = (np.arange(n, dtype=np.int64) % 2) * (1 << 12) + 5  # neighbours differ
    pairs = np.arange(n, dtype=np.int64) // 2 % 9000
    for nb, k in ((2, alternating), (1 << 13, low_equal), (9000, pairs), (4096, (u % np.uint64(4096)).astype(np.int64)),
                  (5000, np.where(u % np.uint64(50) == 0, pairs % 5000, 4999))):
        assert np.array_equal(ctx.call("histogram", ctx.upload(k), nb).numpy(), oracle.histogram(k, nb)), nb
        assert np.array_equal(ctx.call("reduce_into_add_i64", ctx.upload(k), ctx.upload(v), nb).numpy(),
                              oracle.reduce_into_add_i64(k, v, nb)), nb
