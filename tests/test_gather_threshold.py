"""A gather at the turns of its dispatch (k_index.cu, gather_partitions): 7 * 2^22 source rows, and the index
rows from which the partitioned passes run below and from 2^25 source rows."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SMALL, LARGE = 7 << 22, 1 << 25


@pytest.mark.parametrize("source,index", [
    (SMALL - 1, SMALL - 1), (SMALL, SMALL // 2 + 5), (SMALL, SMALL * 3 // 4 - 1), (SMALL, SMALL * 3 // 4),
    (SMALL + 77, SMALL + 77), (LARGE - 1, LARGE // 2 + 9), (LARGE, LARGE // 2), (LARGE, LARGE // 2 - 1)])
def test_rows(ctx, source, index):
    x = ctx.call("rand_f64", source, 5)
    h = oracle.rand_f64(source, 5)
    i = (oracle.rand_i64(index, 6).view(np.uint64) % np.uint64(source)).astype(np.int64)
    assert np.array_equal(ctx.call("gather_f64", x, ctx.upload(i)).numpy(), h[i])
