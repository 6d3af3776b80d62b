"""Canonical f64 sums whose lanes cross binades at the places where the walk (k_canon.cu) changes its way:
in a lane's first tile, in every segment of a tile, on a tile's and a chunk's edge, through several binades
at once, with halfway rows, zeros, subnormals, outliers, infinities, and in a second update from a state that
is not zero. Bit for bit against the oracle."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [4096 * 2, 4096 * 31 + 16, 4096 * 33 + 4080, 4096 * 70 + 5, (1 << 20) + 3]


def rows(kind, n):
    x = oracle.rand_f64(n, n)
    blk = np.arange(n) // 16
    if kind == "uniform":
        return x
    if kind == "ties":  # few bits: halfway rows once the sum has passed 2^40
        return np.floor(x * 8.0) * 2.0**-13 + np.where(blk == 0, 2.0**39, 0.0)
    if kind == "doubling":  # a crossing every few tiles, then every few rows
        return x * 2.0 ** np.minimum((blk // 200) % 60, 50)
    if kind == "jumps":  # several binades within a row
        return np.where(blk % 777 == 776, x * 2.0 ** (blk // 777 % 300 * 3), x)
    if kind == "zeros":
        return np.where(blk % 300 < 290, 0.0, x)
    if kind == "tiny":  # subnormal first, then ordinary
        return np.where(blk < 300, x * 2.0**-1060, np.where(blk < 600, x * 2.0**-300, x))
    if kind == "infinite":
        return np.where(blk == n // 32, np.inf, x)
    if kind == "late":  # the first tile stays far below its last row
        return np.where((blk == 255) | (blk == 8191), 2.0**40 * x, x)
    return np.where(blk % 1000 == 999, -x * 400.0, x)  # some negative rows


@pytest.mark.parametrize("kind", ["uniform", "ties", "doubling", "jumps", "zeros", "tiny", "infinite", "late", "negative"])
def test_walk(ctx, kind):
    for n in SIZES:
        x = rows(kind, n)
        dx = ctx.upload(x)
        want = oracle.reduce_add_f64(x)
        got = ctx.call("reduce_add_f64", dx)
        assert np.float64(got).tobytes() == np.float64(want).tobytes(), n
        half = n // 32 * 16
        r = ctx.reducer("reduce_add_f64")
        r.update(dx.slice(0, half))
        r.update(dx.slice(half, n))
        assert np.float64(r.finish()).tobytes() == np.float64(want).tobytes(), n
        if n < 300_000:
            got = ctx.call("scan_add_f64", dx).numpy()
            assert np.array_equal(got.view(np.uint64), oracle.scan_add_f64(x).view(np.uint64)), n
