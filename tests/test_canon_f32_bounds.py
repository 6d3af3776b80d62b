"""The lower end of a binade in the canonical f32 sums (k_canon32.cu), as tests/test_canon_bounds.py has it
for f64: runs composed as the kernels compose them against IEEE adds, from states at and just above a power
of two, and sums of columns that rise from one and fall back, at the edges of a thread's rows (8 of a lane),
of a warp's (64), of a tile (512) and of a chunk (16384)."""

import numpy as np
import pytest

import oracle

f32 = np.float32
NO_FALL = 1 << 30


def bits(x):
    return int(f32(x).view(np.uint32))


def run(v, code):
    """run32: (d0, d1, mn, mx), or None."""
    e = (code & 0xFF) << 23
    even, odd = np.uint32(e | 0x400000).view(f32), np.uint32(e | 0x400001).view(f32)
    v = -v if code >> 8 else v
    a, b, lo, hi, down = even, odd, even, even, False
    for x in v:
        down |= bool(np.signbit(x))
        a, b = f32(a + x), f32(b + x)
        lo, hi = min(lo, a), max(hi, a)
    if lo < np.uint32(e | 2).view(f32) or hi > np.uint32(e | 0x7FFFFD).view(f32):
        return None
    base = bits(even)
    return (bits(a) - base, bits(b) - base - 1, bits(lo) - base - 1 if down else NO_FALL, bits(hi) - base + 1)


def then(a, b):
    return (a[0] + (b[1] if a[0] & 1 else b[0]), a[1] + (b[0] if a[1] & 1 else b[1]),
            min(a[2], min(a[0], a[1]) + b[2]), max(a[3], max(a[0], a[1]) + b[3]))


def test_composed_runs_move_states_as_ieee_adds_do():
    rng = np.random.default_rng(17)
    applied = near = 0
    for trial in range(6000):
        E = int(rng.choice([1, 100, 127, 150, 253]))
        code = E | (int(rng.integers(0, 2)) << 8)
        m = int(rng.choice([0, 0, 0, 1, 2, 3, 4, 6, 0x7FFFFF, 0x7FFFFC, int(rng.integers(0, 1 << 23))]))
        s = np.uint32((code << 23) | m).view(f32)
        ulp = f32(np.ldexp(1.0, max(E, 1) - 127 - 23))
        total, rows = None, []
        count = int(rng.integers(2, 9))
        rise = int(rng.integers(0, 7))
        halves = float(rng.choice([0.0, 0.5, 1.0, 1.5]))
        for i in range(count):
            v = np.zeros(8, f32)
            if trial % 2:  # rises, then falls back to about where it began, in two rows of one run
                steps = np.zeros(3)
                if i == 0:
                    steps[0] = rise
                elif i == count - 1:
                    steps[1:] = -halves, halves - rise - rng.choice([0.0, 0.0, 0.1, 0.25, 0.4])
                v[[1, 4, 5]] = (steps * ulp).astype(f32) * f32(-1 if code >> 8 else 1)
            else:
                steps = rng.choice([0.0, 0.25, 0.4, 0.5, 1.0, 1.5, 2.5, 3.0, 6.0], 3) * rng.choice([-1, 1, 1], 3)
                v[rng.integers(0, 8, 3)] = (steps * ulp).astype(f32) * f32(-1 if code >> 8 else 1)
            rows.append(v)
            r = run(v, code)
            total = r if total is None else then(total, r)
        S = m | 1 << 23
        if S + total[3] >= 1 << 24 or S + total[2] <= 1 << 23:
            continue
        applied += 1
        near += m < 8
        want = s
        for x in np.concatenate(rows):
            want = f32(want + x)
        assert bits(want) == bits(s) + (total[1] if S & 1 else total[0]), (code, m, rows)
    assert applied > 1500 and near > 700, (applied, near)


PLACES = [(16, 32, 33), (4096 + 7, 4096 + 8, 4096 + 12), (512 + 63, 512 + 64, 512 + 72), (600, 1024, 1025),
          (511, 512, 1024), (16384 + 8, 2 * 16384 - 1, 2 * 16384), (700, 16384 + 700, 16384 + 1300)]
# A rise and two falls, in ulps of the binade above the state.
MOVES = [(3, 0.5, 2.5), (3, 0.5, 2.7), (0, 0.4, 0), (0, 0.25, 0), (1, 1.3, 0), (2, 1.5, 0.7), (2.5, 1.5, 1.0), (5, 5.2, 0),
         (0.5, 0.4, 0.3), (6, 3, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("place", PLACES)
def test_sums_that_fall_back_to_a_power_of_two(ctx, place):
    n = max(70_000, (place[2] + 600) * 16 + 5)
    ones = ctx.upload(np.ones(n, f32))
    for up, down, more in MOVES:
        for first in (2.0**24, -(2.0**24), 1.0, -0.5):
            x = np.zeros(n, f32)
            u = first * 2.0**-23
            x[0], x[place[0] * 16], x[place[1] * 16], x[place[2] * 16] = first, up * u, -down * u, -more * u
            want = oracle.fold("f32", "add", x)
            dx = ctx.upload(x)
            assert ctx.call("reduce_add_f32", dx, raw=True)[2] == want, (up, down, more, first)
            assert ctx.call("dot_f32", dx, ones, raw=True)[2] == want, (up, down, more, first)


@pytest.mark.gpu
def test_small_whole_rows_around_2p24(ctx):
    x = np.zeros(70_000, f32)
    x[0], x[256], x[512], x[528] = 2.0**24, 6.0, -1.0, -5.0
    assert ctx.call("reduce_add_f32", ctx.upload(x)) == 16777215.0
    rng = np.random.default_rng(5)
    for trial in range(20):
        x = np.zeros(200_000, f32)
        x[0] = 2.0**24
        at = rng.integers(1, 200_000 // 16, 400) * 16
        x[at] = rng.integers(-6, 7, 400)
        assert ctx.call("reduce_add_f32", ctx.upload(x), raw=True)[2] == oracle.fold("f32", "add", x), trial
