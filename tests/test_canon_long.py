"""Canonical sums of columns longer than what the walks hold in shared memory: f64 beyond 2^28 rows
(k_canon.cu), f32 beyond 32 chunks in one step, beyond the mixed chunks and beyond the chunks held
(k_canon32.cu); bit for bit against the oracle."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
f32 = np.float32


def test_f64_sums_beyond_the_chunks_held(ctx):
    n = (1 << 28) + (1 << 24) + 4096 * 5 + 7  # the lanes cross 2^23 past the chunks held
    x = ctx.call("rand_f64", n, 7)
    h = oracle.rand_f64(n, 7)
    assert np.float64(ctx.call("reduce_add_f64", x)).tobytes() == np.float64(oracle.reduce_add_f64(h)).tobytes()
    x = ctx.call("sub_f64", x, 0.25)
    h -= 0.25
    assert np.float64(ctx.call("reduce_add_f64", x)).tobytes() == np.float64(oracle.reduce_add_f64(h)).tobytes()


def f32_sum(ctx, x):
    got, want = ctx.call("reduce_add_f32", ctx.upload(x), raw=True)[2], oracle.fold("f32", "add", x)
    assert got == want, (len(x), got, want)


def test_f32_sums_of_many_chunks(ctx):
    n = 1 << 24  # 64 chunks of 2^18 rows
    u = oracle.rand_f64(n, 5).astype(f32)
    f32_sum(ctx, u)
    chunk = np.arange(n) >> 18
    # Large rows at a chunk's middle: binades crossed inside 60 chunks, more than are held tile by tile.
    x = np.where(np.arange(n) % (1 << 18) // 16 == 5000, u * f32(2.0) ** (chunk % 60 + 10).astype(f32), u)
    f32_sum(ctx, x)
    f32_sum(ctx, np.where(chunk % 2 == 0, u - f32(0.5), u).astype(f32))


def test_f32_sums_beyond_the_chunks_held(ctx):
    n = (1 << 28) + (1 << 22) + 77
    x = oracle.rand_f64(n, 9).astype(f32)
    x[: 1 << 23] *= f32(2.0**-12)
    f32_sum(ctx, x)
