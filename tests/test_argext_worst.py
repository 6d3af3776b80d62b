"""The first extreme of integer rows that are all the worst value: row 0."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {"i64": np.int64, "u64": np.uint64, "i32": np.int32, "u8": np.uint8}


@pytest.mark.parametrize("t", ["i64", "u64", "i32", "u8"])
def test_worst_everywhere(ctx, t):
    info = np.iinfo(DT[t])
    for n in (1, 15, 100_003):
        assert ctx.call("argmin_" + t, ctx.upload(np.full(n, info.max, DT[t]))) == 0
        assert ctx.call("argmax_" + t, ctx.upload(np.full(n, info.min, DT[t]))) == 0
