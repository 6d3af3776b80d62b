"""Reducers and scanners whose updates are captured in a graph: every replay goes on from the state that it
finds, also the first one, and a capture alone feeds no rows."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TYPES = {"f64": np.float64, "i64": np.int64, "f32": np.float32, "i32": np.int32, "u8": np.uint8, "u64": np.uint64}
REDUCERS = ["count_gt_f64", "reduce_add_i64", "reduce_min_f64", "argmax_f64", "reduce_max_i64", "argmin_i64", "reduce_add_f64",
            "dot_f64", "reduce_add_f32", "sumsq_f32", "reduce_add_i32", "reduce_max_i32", "argmin_u8", "reduce_mul_f64",
            "reduce_xor_u64", "count_lt_i32"]
SCANNERS = ["scan_add_i64", "scan_max_f64", "scan_min_f32", "scan_add_i32", "scan_xor_u8", "scan_mul_u64", "scan_by_add_i64",
            "scan_by_min_i64", "scan_by_max_f64"]


def column(t, n, seed):
    x = oracle.rand_f64(n, seed) - 0.25
    return (x if t[0] == "f" else np.abs(x) * 100).astype(TYPES[t])


def args_of(name, a):
    t = name.rsplit("_", 1)[1]
    if name.startswith("count"):
        import verkehrt_gb300 as vk

        return a, vk.Scalar(t, 0.25 if t[0] == "f" else 25)
    return (a, a) if name.startswith("dot") else (a,)


@pytest.mark.parametrize("name", REDUCERS)
@pytest.mark.parametrize("n", [1600, 98_304])
def test_replays_of_a_captured_update(ctx, name, n):
    t = name.rsplit("_", 1)[1]
    a, b, c = (column(t, n, s) for s in (1, 2, 3))
    da, db, dc = ctx.upload(a), ctx.upload(b), ctx.upload(c)

    def want(*parts):
        return ctx.call(name, *args_of(name, ctx.upload(np.concatenate(parts))), raw=True)[2]

    want(a, b, b, c, b)  # sizes the scratch arena
    # The reducer's first update is the captured one.
    r = ctx.reducer(name)
    ctx.synchronize()
    ctx.graph_begin()
    r.update(*args_of(name, db))
    g = ctx.graph_end()
    for _ in range(3):
        g.launch()
    assert r.finish(raw=True)[2] == want(b, b, b)
    # Others around it.
    r = ctx.reducer(name)
    r.update(*args_of(name, da))
    ctx.synchronize()
    ctx.graph_begin()
    r.update(*args_of(name, db))
    g = ctx.graph_end()
    g.launch()
    g.launch()
    other = ctx.call(name, *args_of(name, dc), raw=True)[2]
    assert other == want(c)
    if not name.startswith("arg"):  # a replayed update numbers its rows as it did when it was captured
        r.update(*args_of(name, dc))
        g.launch()
        assert r.finish(raw=True)[2] == want(a, b, b, c, b)


@pytest.mark.parametrize("name", REDUCERS)
def test_a_capture_feeds_no_rows(ctx, name):
    t = name.rsplit("_", 1)[1]
    db = ctx.upload(column(t, 1600, 2))
    ctx.call(name, *args_of(name, db))  # leaves its result in a slot
    r = ctx.reducer(name)
    ctx.synchronize()
    ctx.graph_begin()
    r.update(*args_of(name, db))
    g = ctx.graph_end()
    if "min" in name or "max" in name:
        with pytest.raises(Exception, match="empty array"):
            r.finish()
    else:
        assert r.finish() == (1.0 if "mul" in name else 0)
    del g


@pytest.mark.parametrize("name", SCANNERS)
def test_replays_of_a_captured_scan(ctx, name):
    n = 5000
    t = name.rsplit("_", 1)[1]
    x = column(t, n, 4)
    by = name.startswith("scan_by")
    starts = oracle.rand_f64(n, 5) < 0.01
    starts[:100] = False
    dx = ctx.upload(x)
    extra = (ctx.upload(starts),) if by else ()
    three = ctx.call(name, ctx.upload(np.tile(x, 3)), *((ctx.upload(np.tile(starts, 3)),) if by else ()))
    want = three.numpy()
    out = ctx.new_array(three.type, n)
    warm = ctx.scanner(name)
    warm.update((dx,) + extra, out)
    s = ctx.scanner(name)
    ctx.synchronize()
    ctx.graph_begin()
    s.update((dx,) + extra, out)
    g = ctx.graph_end()
    for k in range(3):
        g.launch()
        assert np.array_equal(out.numpy(), want[k * n:(k + 1) * n]), k
