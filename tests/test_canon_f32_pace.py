"""Canonical f32 sums whose lanes leave their binade all the time (k_canon32.cu): the walk's tiles end as
chains; bit for bit against the oracle, from columns where some tiles do to columns where all do, and in a time
that does not run away from an ordinary column's."""

import time

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
f32 = np.float32


def column(kind, n):
    u = oracle.rand_f64(n, 3)
    sign = (np.arange(n) // 16 % 2) * 2.0 - 1.0
    if kind == "alternating":
        return (sign * (u + 1.0) * 1e6).astype(f32)
    if kind == "stretches":  # alternating for a third of every 20,000 rows
        return np.where(np.arange(n) // 7000 % 3 == 1, sign * (u + 1.0) * 1e6, u).astype(f32)
    if kind == "specials":
        x = (sign * (u + 1.0) * 1e6).astype(f32)
        x[n // 2] = np.inf
        return x
    if kind == "overflow":
        with np.errstate(over="ignore"):
            return (sign * (u + 1.0) * 1.6e38 + 1e38).astype(f32)
    return (u - 0.5).astype(f32)


@pytest.mark.parametrize("kind", ["alternating", "stretches", "specials", "overflow", "centred"])
def test_sums_equal_the_oracle(ctx, kind):
    for n in (70_000, 8192 * 24 + 16 * 100 + 3, 700_001):
        x = column(kind, n)
        want, got = oracle.fold("f32", "add", x), ctx.call("reduce_add_f32", ctx.upload(x), raw=True)[2]
        w, g = np.uint32(want & 0xFFFFFFFF), np.uint32(got & 0xFFFFFFFF)
        assert w == g or (np.isnan(w.view(f32)) and np.isnan(g.view(f32))), n


@pytest.mark.parametrize("n", [1 << 17, 1 << 20])
def test_time_of_a_column_that_wanders(ctx, n):
    def best(kind):
        dx, t = ctx.upload(column(kind, n) if kind != "uniform" else oracle.rand_f64(n, 1).astype(f32)), []
        for _ in range(6):
            ctx.synchronize()
            t0 = time.perf_counter()
            ctx.call("reduce_add_f32", dx)
            t.append(time.perf_counter() - t0)
        return min(t)

    uniform, wandering = best("uniform"), best("alternating")
    limit = 3.5 if n == 1 << 17 else 12  # 5.2 and 25 times without chains
    assert wandering < limit * uniform, (wandering, uniform)
