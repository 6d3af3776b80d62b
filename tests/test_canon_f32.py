"""The canonical f32 sums (k_canon32.cu) bit for bit against the oracle at the edges of their tiles
(8192 rows), chunks (32 tiles) and of the short path (2^16 rows), on rows that wander around zero,
tie, cross many binades or hold special values; and the rule they rest on, that a run of rows moves
every state of a binade by the ulps it moves 1.5 * 2^E and the next float, against IEEE adds."""

import numpy as np
import pytest

import oracle

f32 = np.float32


def rows(kind, n, seed):
    u = oracle.rand_f64(n, seed)
    r = oracle.rand_i64(n, seed + 1)
    if kind == "uniform":
        return u.astype(f32)
    if kind == "centred":
        return (u - 0.5).astype(f32)
    if kind == "negative":
        return (-u).astype(f32)
    if kind == "ties":  # quarters: most adds of a large sum are halfway, of either sign
        return ((r % 9 - 3) * 0.25).astype(f32)
    if kind == "up_ties":
        return ((r % 7 + 7) % 7 * 0.5).astype(f32)
    if kind == "wide":
        return np.ldexp((u - 0.25), (r % 40).astype(np.int32)).astype(f32)
    if kind == "zeros":
        x = np.zeros(n, f32)
        x[n // 2:] = u[n // 2:]
        return x
    if kind == "stalls":  # a large row early: the later ones are far below half an ulp
        x = u.astype(f32)
        x[min(n - 1, 40)] = 3e9
        return x
    x = (u - 0.25).astype(f32)
    x[n // 3] = np.inf if kind == "inf" else np.nan
    return x


KINDS = ["uniform", "centred", "negative", "ties", "up_ties", "wide", "zeros", "stalls", "inf", "nan"]


def same(got, want):
    g, w = np.uint32(got & 0xFFFFFFFF), np.uint32(want & 0xFFFFFFFF)
    return g == w or (np.isnan(g.view(f32)) and np.isnan(w.view(f32)))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_sums_equal_the_oracle(ctx, kind):
    import verkehrt_gb300 as vk

    for n in (3, 4097, (1 << 16) - 1, (1 << 16) + 16, (1 << 16) + 8191, 32 * 8192, 32 * 8192 + 17, 1_000_003):
        x, y = rows(kind, n, n), rows("uniform", n, n + 9)
        dx, dy = ctx.upload(x), ctx.upload(y)
        assert same(ctx.call("reduce_add_f32", dx, raw=True)[2], oracle.fold("f32", "add", x)), n
        assert same(ctx.call("dot_f32", dx, dy, raw=True)[2], oracle.fused_sum("f32", "dot", x, y)), n
        if n > (1 << 16):
            assert same(ctx.call("sumsq_f32", dx, raw=True)[2], oracle.fused_sum("f32", "sumsq", x)), n
            got = ctx.call("condsum_gt_f32", dx, vk.Scalar("f32", 0.25), vk.Scalar("f32", -0.125), raw=True)[2]
            assert same(got, oracle.fused_sum("f32", "condsum", x, cmp="gt", c=0.25, e=-0.125)), n
            # A slice off the 16-byte grid, and the same rows in two updates.
            assert same(ctx.call("reduce_add_f32", dx.slice(3, n), raw=True)[2], oracle.fold("f32", "add", x[3:])), n
            r = ctx.reducer("reduce_add_f32")
            r.update(dx.slice(0, 40_000))
            r.update(dx.slice(40_000, n))
            assert same(r.finish(raw=True)[2], oracle.fold("f32", "add", x)), n


def bits(x):
    return int(f32(x).view(np.uint32))


def run(v, code):
    """run32: (d0, d1, mn, mx), or None."""
    e = (code & 0xFF) << 23
    even, odd = np.uint32(e | 0x400000).view(f32), np.uint32(e | 0x400001).view(f32)
    lo_ok, hi_ok = np.uint32(e | 2).view(f32), np.uint32(e | 0x7FFFFD).view(f32)
    v = -v if code >> 8 else v
    a, b, lo, hi, down = even, odd, even, even, False
    for x in v:
        down |= bool(np.signbit(x))
        a, b = f32(a + x), f32(b + x)
        lo, hi = min(lo, a), max(hi, a)
    if not (lo >= lo_ok and hi <= hi_ok):
        return None
    base = bits(even)
    return bits(a) - base, bits(b) - base - 1, bits(lo) - base - 1 if down else 0, bits(hi) - base + 1


def then(a, b):
    return (a[0] + (b[1] if a[0] & 1 else b[0]), a[1] + (b[0] if a[1] & 1 else b[1]),
            min(a[2], min(a[0], a[1]) + b[2]), max(a[3], max(a[0], a[1]) + b[3]))


def test_runs_move_states_as_ieee_adds_do():
    rng = np.random.default_rng(3)
    applied = 0
    for trial in range(4000):
        E = int(rng.integers(1, 254)) if trial % 4 == 0 else 127
        code = E | (int(rng.integers(0, 2)) << 8)
        # States at the ends of the binade and inside it, both parities.
        m = int(rng.choice([0, 1, 2, 3, 0x7FFFFF, 0x7FFFFE, 0x7FFFFC, 0x400000, int(rng.integers(0, 1 << 23))]))
        s = np.uint32((code << 23) | m).view(f32)
        ulp = np.ldexp(1.0, E - 127 - 23)
        scale = [0.5, 0.25, 1.0, 0.3, 3.7][trial % 5] * ulp
        v = (rng.integers(-3 if trial % 3 else 0, 6, 16) * scale).astype(f32)
        f, g = run(v[:8], code), run(v[8:], code)
        if f is None or g is None:
            continue
        f = then(f, g)
        S = (bits(s) & 0x7FFFFF) | 0x800000
        if S + f[3] >= 1 << 24 or (f[2] < 0 and S + f[2] <= 1 << 23):
            continue
        applied += 1
        want = s
        for x in v:
            want = f32(want + x)
        assert bits(want) == bits(s) + (f[1] if S & 1 else f[0]), (code, m, v)
    assert applied > 1000
