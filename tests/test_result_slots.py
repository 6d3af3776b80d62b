"""Reducers whose results kernels write in place (reduce_common.h): more of them at once than there are
slots, dropped unfinished, finished without rows, and inside a captured graph while others run; and
selections of few rows (k_select.cu) at the edges of their one-block form."""

import numpy as np
import pytest

import oracle
from helpers import with_specials

pytestmark = pytest.mark.gpu

NAMES = ["count_gt_f64", "reduce_add_i64", "reduce_min_f64", "argmax_f64", "reduce_add_f64", "reduce_add_f32",
         "reduce_max_i32", "argmin_u8", "reduce_mul_f64"]
TYPES = {"f64": np.float64, "i64": np.int64, "f32": np.float32, "i32": np.int32, "u8": np.uint8}


def column(name, n, seed):
    t = name.rsplit("_", 1)[1]
    x = oracle.rand_f64(n, seed) - 0.25
    return (x if t[0] == "f" else np.abs(x) * 100).astype(TYPES[t])


def args_of(name, a):
    return (a, 0.25) if name.startswith("count") else (a,)


def test_many_reducers_at_once(ctx):
    cols = {name: [ctx.upload(column(name, 3000, 7 * i)) for i in range(12)] for name in NAMES}
    live = [(name, a, ctx.reducer(name)) for name in NAMES for a in cols[name]]  # more than the slots
    for name, a, r in live:
        r.update(*args_of(name, a.slice(0, 1600)))
    dropped = [ctx.reducer("reduce_add_f64") for _ in range(5)]
    for d in dropped:
        d.update(cols["reduce_add_f64"][0])
    del dropped, d
    for name, a, r in reversed(live):
        r.update(*args_of(name, a.slice(1600, 3000)))
        assert r.finish(raw=True)[2] == ctx.call(name, *args_of(name, a), raw=True)[2], name
    for name in NAMES:
        r = ctx.reducer(name)
        if "min" in name or "max" in name:
            with pytest.raises(Exception, match="empty array"):
                r.finish()
        else:
            assert r.finish() == (1.0 if "mul" in name else 0), name


def test_captured_reductions_between_calls(ctx):
    cols = {name: ctx.upload(column(name, 5000, 3)) for name in NAMES}
    outs = {}
    for name in NAMES:
        t = ctx.call(name, *args_of(name, cols[name]), raw=True)[0]
        outs[name] = ctx.new_array(t, 1)
        ctx.call_into(name, *args_of(name, cols[name]), out=outs[name])
    ctx.synchronize()
    ctx.graph_begin()
    for name in NAMES:
        ctx.call_into(name, *args_of(name, cols[name]), out=outs[name])
    g = ctx.graph_end()
    want = {name: ctx.call(name, *args_of(name, cols[name])) for name in NAMES}
    for _ in range(3):
        g.launch()
        for name in NAMES:  # calls of their own between the replays
            assert ctx.call(name, *args_of(name, cols[name])) == want[name], name
    for name in NAMES:
        assert outs[name].numpy()[0] == want[name], name


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 16383, 16384, 16385])
def test_selections_of_few_rows(ctx, n):
    x = with_specials(n, n)
    dx = ctx.upload(x)
    for cmp, c in (("gt", 0.5), ("ne", 0.0), ("le", np.inf), ("eq", np.nan), ("lt", -1e300)):
        got = ctx.call("filter_%s_f64" % cmp, dx, c).numpy()
        assert np.array_equal(got.view(np.uint64), oracle.filter_cmp_f64(x, cmp, c).view(np.uint64)), (cmp, c)
    for keep in (0.0, 0.03, 0.5, 1.0):
        m = oracle.rand_f64(n, 5) < keep
        dm = ctx.upload(m)
        assert np.array_equal(ctx.call("where", dm).numpy(), np.flatnonzero(m))
        for t in ("f64", "i32", "u8"):
            v = (oracle.rand_f64(n, 6) * 200).astype(oracle.NP_TYPES[t])
            assert np.array_equal(ctx.call("compress_" + t, ctx.upload(v), dm).numpy(), v[m]), t
            if n > 3:
                got = ctx.call("compress_" + t, ctx.upload(v).slice(1, n), dm.slice(1, n)).numpy()
                assert np.array_equal(got, v[1:][m[1:]]), t
