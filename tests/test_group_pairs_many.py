"""group_id2 where the first table gives up (more than 2^20 distinct pairs, or many in a few slots) and the full
table is numbered: sizes about the numbering's tiles, pairs that repeat near and far."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 20) + 4097, 1 << 22, (1 << 22) + 1, (1 << 22) + 4095])
@pytest.mark.parametrize("distinct", ["all", "half", "near"])
def test_many_pairs(ctx, n, distinct):
    a = oracle.rand_i64(n, 11)
    if distinct == "half":
        a[n // 2 :] = a[: n - n // 2]
    elif distinct == "near":  # each pair twice, in neighbouring rows
        a = np.repeat(a[: n - n // 2], 2)[:n]
    b = a % 7 - 3
    _, first, inverse = np.unique(a, return_index=True, return_inverse=True)
    rank = np.empty(len(first), np.int64)
    rank[np.argsort(first)] = np.arange(len(first))
    got = ctx.call("group_id2_i64_i64", ctx.upload(a), ctx.upload(b)).numpy()
    assert np.array_equal(got, rank[inverse.reshape(-1)])
