"""reduce_into_add_f64 of uneven key columns (k_reduce_into_f64.cu): most rows in one bucket, in a few, or each
bucket's rows in one of the sixteen stripes, so that chains are far longer than even keys'; bit for bit against
the oracle, and no slower for it than a few masked sums."""

import time

import numpy as np
import pytest

import oracle
from helpers import varied

pytestmark = pytest.mark.gpu


def keys_of(kind, n, nb):
    u = oracle.rand_i64(n, 7).view(np.uint64)
    even = (u % np.uint64(nb)).astype(np.int64)
    hot = u >> np.uint64(32) < np.uint64(0xF3333333)  # 95% of the rows
    if kind == "even":
        return even
    if kind == "one":
        return np.where(hot, nb - 1, even)
    if kind == "all":
        return np.full(n, nb // 2)
    if kind == "few":
        return np.where(hot, even % min(nb, 3) * (nb // min(nb, 3)), even)
    if kind == "many":  # more long chains than masked sums pay for
        return np.where(hot, even % min(nb, 40), even)
    return np.arange(n) % nb  # "stripes"


@pytest.mark.parametrize("kind", ["one", "all", "few", "many", "stripes"])
@pytest.mark.parametrize("nb", [8, 16, 17, 300, 70_000, 1 << 20])
def test_uneven_keys(ctx, kind, nb):
    for n in (65_551, 1_000_000, 2_000_003):
        x = varied(n, 3) if kind != "few" else oracle.rand_f64(n, 3)
        k = keys_of(kind, n, nb)
        k[-3:] = (0, nb - 1, nb // 2)
        got = ctx.call("reduce_into_add_f64", ctx.upload(k), ctx.upload(x), nb).numpy()
        assert np.array_equal(got.view(np.uint64), oracle.reduce_into_add_f64(k, x, nb).view(np.uint64)), n


def test_more_long_chains_than_are_noted(ctx):
    n, nb = 4_000_007, 100_000
    k = np.arange(n) // 4000 * 97 % nb  # a thousand buckets of 250-row chains
    k[: n // 2] = np.arange(n // 2) % 300 * 16
    x = oracle.rand_f64(n, 5)
    got = ctx.call("reduce_into_add_f64", ctx.upload(k), ctx.upload(x), nb).numpy()
    assert np.array_equal(got.view(np.uint64), oracle.reduce_into_add_f64(k, x, nb).view(np.uint64))


@pytest.mark.parametrize("nb", [16, 1024])
def test_time_of_a_skewed_column(ctx, nb):
    n = 1 << 22
    x = ctx.upload(oracle.rand_f64(n, 1))

    def best(k):
        dk, t = ctx.upload(k), []
        for _ in range(4):
            ctx.synchronize()
            t0 = time.perf_counter()
            ctx.call("reduce_into_add_f64", dk, x, nb)
            t.append(time.perf_counter() - t0)
        return min(t)

    even, skewed = best(keys_of("even", n, nb)), best(keys_of("one", n, nb))
    assert skewed < 6 * even, (skewed, even)  # one masked sum beside the even column's time; chains: 13 and 70 times
