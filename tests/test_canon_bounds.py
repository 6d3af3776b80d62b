"""The lower end of a binade in the canonical f64 sums (k_canon.cu). A lane's state moves over a run of rows
by whole ulps of its binade 2^E, which holds only while every exact sum on the way lies in it: a fall that
rounds to 2^E, or to no ulp at all from there, may round below it, whatever rose before. The composition of
moves against IEEE adds, and sums and scans of columns that rise from a power of two and fall back to it,
with the rise and the fall in one segment (8 rows of a lane), tile (256) or chunk (8192) or in several."""

from fractions import Fraction

import numpy as np
import pytest

import oracle

ONE = 1 << 52
NO_FALL = 1 << 61


# ---------------------------------------------------------------- the rule, restated


def nearest(q):
    """(the nearest whole number, to even; whether q is halfway)."""
    f = q.numerator // q.denominator
    r = q - f
    if r == Fraction(1, 2):
        return f + (f & 1), True
    return f + (r > Fraction(1, 2)), False


def segment(v, E):
    """seg_tf: (up, down, falls) of rows of either sign, or (d0, d1) of rows without a negative one."""
    u = Fraction(2) ** (E - 52)
    if any(abs(x) >= 2.0**E for x in v):
        return None
    if any(x < 0 for x in v):
        up = down = 0
        for x in v:
            inc, tie = nearest(Fraction(abs(x)) / u)
            if tie:
                return None
            up, down = (up + inc, down) if x > 0 else (up, down + inc)
        return up, down, True
    d = [0, 0]
    for x in v:
        q = Fraction(x) / u
        f = q.numerator // q.denominator
        half = q - f == Fraction(1, 2)
        for p in (0, 1):
            d[p] += f + ((p + d[p] + f) & 1) if half else nearest(q)[0]
    return d[0], d[1], False


def move(f, neg):
    """A function as (d0, d1, mn, mx) of the state's magnitude, or None where it does not apply."""
    if f[2]:
        up, down, _ = f
        return (down - up, down - up, -up, down) if neg else (up - down, up - down, -down, up)
    if f[0] != f[1]:
        return None if neg else (f[0], f[1], NO_FALL, max(f[0], f[1]))
    return (-f[0], -f[0], -f[0], 0) if neg else (f[0], f[0], NO_FALL, f[0])


def then(a, b):
    return (a[0] + (b[1] if a[0] & 1 else b[0]), a[1] + (b[0] if a[1] & 1 else b[1]),
            min(a[2], min(a[0], a[1]) + b[2]), max(a[3], max(a[0], a[1]) + b[3]))


def carried(S, m):
    return S + m[3] < 2 * ONE and S + m[2] > ONE


def test_moves_are_those_of_ieee_adds():
    rng = np.random.default_rng(11)
    applied = near = 0
    for trial in range(12000):
        E = int(rng.choice([0, -40, 100]))
        u = 2.0 ** (E - 52)
        S = ONE + int(rng.choice([0, 0, 0, 1, 2, 3, 5, ONE - 2, ONE - 1, int(rng.integers(0, ONE))]))
        neg = bool(rng.integers(0, 2))
        runs, total = [], None
        for _ in range(int(rng.integers(2, 9))):
            v = np.zeros(8)
            at = rng.integers(0, 8, 3)
            v[at] = rng.choice([0.0, 0.2, 0.25, 0.3, 0.4, 0.5, 1.0, 1.4, 2.0, 2.5, 5.0, 6.0], 3) * rng.choice([-1, 1], 3) * u
            runs.append(v)
            f = segment(v, E)
            m = None if f is None else move(f, neg)
            if m is None:
                total = None
                break
            total = m if total is None else then(total, m)
        if total is None or not carried(S, total):
            continue
        applied += 1
        near += S - ONE < 6
        s = (-1.0 if neg else 1.0) * S * u
        want = s
        for x in np.concatenate(runs):
            want = want + x
        got = (-1.0 if neg else 1.0) * (S + total[S & 1]) * u
        assert got == want, (E, S - ONE, neg, runs)
    assert applied > 500 and near > 200, (applied, near)


# ---------------------------------------------------------------- sums and scans


# Rows of lane 0 (a block is 16 rows) at which the column rises and falls; 256 a tile, 8192 a chunk.
PLACES = [(8, 16), (256 + 3, 256 + 4), (256 + 8, 256 + 16), (256 + 250, 512), (8 * 256, 20 * 256 + 77), (8191, 8192),
          (8192 + 8, 16384 + 300)]
# The rise and the fall in ulps of the binade above the state.
MOVES = [(0, 0.4), (0, 0.26), (0, 0.25), (0, 0.2), (1, 1.4), (1, 1.26), (1, 1.0), (3, 3.3), (2.5, 2.4), (0.5, 0.4), (1, 2.0),
         (7, 7.2)]


def column(first, place, up, down, n):
    x = np.zeros(n)
    u = 2.0**-52 * first
    x[0] = first
    x[place[0] * 16] = up * u
    x[place[1] * 16] = -down * u
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("place", PLACES)
def test_sums_that_fall_back_to_a_power_of_two(ctx, place):
    n = max(8192, (place[1] + 300) * 16)
    ones = ctx.upload(np.ones(n))
    for up, down in MOVES:
        for sign in (1.0, -1.0):
            x = sign * column(4.0, place, up, down, n)
            want = np.float64(oracle.reduce_add_f64(x)).tobytes()
            dx = ctx.upload(x)
            assert np.float64(ctx.call("reduce_add_f64", dx)).tobytes() == want, (up, down, sign)
            assert np.float64(ctx.call("dot_f64", dx, ones)).tobytes() == want, (up, down, sign)
            assert np.float64(ctx.call("condsum_ne_f64", dx, 9.0, 0.0)).tobytes() == want, (up, down, sign)
            got = ctx.call("scan_add_f64", dx).numpy()
            assert np.array_equal(got.view(np.uint64), oracle.scan_add_f64(x).view(np.uint64)), (up, down, sign)


@pytest.mark.gpu
def test_sum_that_rises_an_ulp_and_falls_below_one(ctx):
    x = np.zeros(8192)
    x[0], x[128], x[256] = 1.0, 2.0**-52, -1.4 * 2.0**-52
    assert ctx.call("reduce_add_f64", ctx.upload(x)) == 0.9999999999999999


@pytest.mark.gpu
def test_columns_of_zeros_behind_a_power_of_two(ctx):
    for n in (100_000, 1 << 20):
        for first in (-1.0, 1.0, -0.375):
            for zero in (0.0, -0.0):
                x = np.full(n, zero)
                x[::997] = first
                x[n - 40] = first * 0.3
                got = ctx.call("reduce_add_f64", ctx.upload(x))
                assert np.float64(got).tobytes() == np.float64(oracle.reduce_add_f64(x)).tobytes(), (n, first, zero)
                x[17:] = zero
                x[n - 30] = -first * 2.0**-54 * 1.7
                got = ctx.call("reduce_add_f64", ctx.upload(x))
                assert np.float64(got).tobytes() == np.float64(oracle.reduce_add_f64(x)).tobytes(), (n, first, zero)
