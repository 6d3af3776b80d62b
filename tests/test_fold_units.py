"""Order-free folds and first extremes of every width (k_families.cu, k_reduce.cu) around their 16-byte units:
rows on and off the grid, and columns that lie differently on it."""

import numpy as np
import pytest

import oracle
import verkehrt_gb300 as vk

pytestmark = pytest.mark.gpu

DT = {"f32": np.float32, "i64": np.int64, "u64": np.uint64, "i32": np.int32, "u8": np.uint8}


@pytest.mark.parametrize("t", list(DT))
def test_units(ctx, t):
    for n in (1, 3, 16, 17, 1000, 300_001):
        for ox, oy in ((0, 0), (1, 1), (3, 0)):
            x = (oracle.rand_i64(n + 3, n) >> 20).astype(DT[t])
            y = (oracle.rand_i64(n + 3, 5) >> 20).astype(DT[t])
            dx, dy = ctx.upload(x).slice(ox, ox + n), ctx.upload(y).slice(oy, oy + n)
            x, y = x[ox:ox + n], y[oy:oy + n]
            assert ctx.call("argmin_" + t, dx) == int(np.argmin(x))
            assert ctx.call("argmax_" + t, dx) == int(np.argmax(x))
            assert ctx.call("reduce_max_" + t, dx) == x.max()
            if t == "f32":
                assert ctx.call("count_gt_f32", dx, vk.Scalar("f32", 0.0)) == int((x > 0).sum())
                continue
            wide = np.uint64 if t in ("u64", "u8") else np.int64
            assert ctx.call("reduce_add_" + t, dx) == x.sum(dtype=wide)
            assert ctx.call("reduce_xor_" + t, dx) == np.bitwise_xor.reduce(x)
            if t != "u8":
                assert ctx.call("dot_" + t, dx, dy) == (x * y).astype(wide).sum(dtype=wide)
