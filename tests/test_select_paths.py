"""Selections of every kind and width (k_select.cu) at the edges of steps, slices and tiles, on rows off the
16-byte grid, in both tile sizes, and filters' ranges at their ends: zeros of both signs, infinities, NaNs,
the least and greatest integers. Bit for bit against the oracle."""

import numpy as np
import pytest

import oracle
import verkehrt_gb300 as vk

pytestmark = pytest.mark.gpu

DT = {"f64": np.float64, "f32": np.float32, "i64": np.int64, "u64": np.uint64, "i32": np.int32}
SIZES = [1, 31, 16_385, 8192 * 3, 8192 * 3 + 15, 8192 * 3 + 16, 8192 * 5 + 33, 70_001]
BIG = 152 * 2 * 512 * 64 + 12_345  # past the larger tiles' rule on any width


def values(t, n):
    u = oracle.rand_i64(n, n + 5).view(np.uint64)
    if t in ("f64", "f32"):
        x = ((u >> np.uint64(40)).astype(np.int64) - (1 << 23)).astype(DT[t]) / DT[t](1 << 20)
        ends = [0.0, -0.0, np.inf, -np.inf, np.nan, 1.0]
    else:
        x = (u >> np.uint64(3)).astype(DT[t]) if t != "i32" else u.astype(np.uint32).view(np.int32).copy()
        info = np.iinfo(DT[t])
        ends = [info.min, info.max, 0, 1]
    for i, e in enumerate(ends):
        x[i::37] = e
    return x


def constants(t):
    if t in ("f64", "f32"):
        return [0.0, -0.0, 1.0, -1.5, np.inf, -np.inf, np.nan]
    info = np.iinfo(DT[t])
    return [info.min, info.max, 0, 1, info.max // 2]


def same(a, b):
    return a.dtype == b.dtype and np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("t", list(DT))
def test_filters(ctx, t):
    for n in SIZES:
        x = values(t, n)
        for off in (0, 1):
            dx = ctx.upload(np.concatenate([x[:off], x])).slice(off, off + n)
            for c in constants(t) if n in (31, 70_001) else constants(t)[-2:]:
                with np.errstate(invalid="ignore"):
                    k = DT[t](c)
                    masks = {"eq": x == k, "ne": x != k, "lt": x < k, "le": x <= k, "gt": x > k, "ge": x >= k}
                for cmp, m in masks.items():
                    got = ctx.call("filter_%s_%s" % (cmp, t), dx, vk.Scalar(t, c)).numpy()
                    assert same(got, x[m]), (n, off, cmp, c)


def test_masks(ctx):
    for n in SIZES + [BIG]:
        m = oracle.rand_i64(n, n) % 3 == 0
        m[::1000] = True
        for off in (0, 1, 3) if n < BIG else (0, 5):
            dm = ctx.upload(np.concatenate([np.ones(off, m.dtype), m])).slice(off, off + n)
            assert same(ctx.call("where", dm).numpy(), np.flatnonzero(m).astype(np.int64)), (n, off)
            for t in ("i64", "f32", "u8") if n < BIG else ("f32", "u8"):
                v = oracle.rand_i64(n, 3).astype({"i64": np.int64, "f32": np.float32, "u8": np.uint8}[t])
                dv = ctx.upload(np.concatenate([np.ones(off, v.dtype), v])).slice(off, off + n)
                assert same(ctx.call("compress_" + t, dv, dm).numpy(), v[m]), (n, off, t)


def test_large_filter(ctx):
    x = (oracle.rand_i64(BIG, 9) >> 40).astype(np.float32)
    x[::101] = np.nan
    with np.errstate(invalid="ignore"):
        want = x[x > -5.0]
    assert same(ctx.call("filter_gt_f32", ctx.upload(x), vk.Scalar("f32", -5.0)).numpy(), want)
