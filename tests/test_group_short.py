"""group_id of inputs whose first table is the full one (k_group.cu, gi_insert_short_kernel), where each block
takes the way of few or of many keys by its first rows: columns of either sort and of both, blocks that decide
by rows unlike the rest, the free slot's own key, and pairs."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

FREE = np.uint64(0x8080808080808080).astype(np.int64)  # the key that a free slot holds


def column(kind, n):
    r = oracle.rand_i64(n, 3)
    i = np.arange(n)
    if kind == "distinct":
        return r
    if kind == "few":
        return r % 10
    if kind == "blocks":  # one block's rows distinct, the next one's few
        return np.where(i // 1024 % 2 == 0, r, r % 3)
    if kind == "first rows apart":  # each block's first 256 rows are distinct, the others few
        return np.where(i % 1024 < 256, r % 65536 * 65536 + i, r % 5)
    k = r % 40_000
    k[r % 7 == 0] = FREE
    return k


@pytest.mark.parametrize("kind", ["distinct", "few", "blocks", "first rows apart", "free"])
@pytest.mark.parametrize("n", [1, 31, 1025, 32 * 1024 - 1, 32 * 1024 + 1, 200_003, 1 << 20])
def test_ids(ctx, kind, n):
    k = column(kind, n)
    dk = ctx.upload(k)
    assert np.array_equal(ctx.call("group_id_i64", dk).numpy(), oracle.group_id_i64(k))
    b = np.where(oracle.rand_i64(n, 5) % 3 == 0, FREE, k % 7)
    _, first, inverse = np.unique(np.stack([k, b], 1), axis=0, return_index=True, return_inverse=True)
    rank = np.empty(len(first), np.int64)
    rank[np.argsort(first)] = np.arange(len(first))
    got = ctx.call("group_id2_i64_i64", dk, ctx.upload(b)).numpy()
    assert np.array_equal(got, rank[inverse.reshape(-1)])
