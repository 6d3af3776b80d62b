"""The calls that a program of the array language makes on the `cuda` kernel table, with their sizes.

`listed()` names twelve of them, `draw(rng)` gives further ones of the same ranges. `prepare` makes
what the program has in hand (device arrays), `run` is one pass through the package's public entry
points, `exact` its float results in 64 bits from torch alone, and `work` the bytes and operations
that a pass cannot do without.

The kinds of case, and what each stands for:

  program    the README program, sum(x*y), count(x > 0.5), length(filter(x, 0.99)): a request of a
             few statements, where latency and launches count (with `graph`, the statements whose
             results stay on the device, captured once and replayed)
  reduce     the summary of a column: sum, dot, min, max, argmin, argmax and a count
  narrow     the summary of a 32-bit column (f32 measurements, i32 codes), and a filter of it
  select     the rows above a threshold, the rows of a mask, and the row numbers of a mask
  gather     a column read by row numbers (a join or a permutation)
  scan       a running fold over a column, and the same within segments: i64 and i32 sums, the
             running maximum of an f64 column
  fsum       float sums that keep the language's order: running, running within segments, and per
             bucket
  sort       the stable order of a key column, and another column put into that order
  group      group numbers of a key column, the number of groups, a sum and a count per group
  batch      many short arrays that run one statement each: kept sums, counts and orders
  expr       elementwise expressions evaluated as regions: an array result and two folds
"""

import math

import numpy as np
import torch

import verkehrt_gb300 as vk

_DEVICE = "cuda"
_TORCH = {"f64": torch.float64, "f32": torch.float32, "i64": torch.int64, "i32": torch.int32,
          "u8": torch.uint8, "bool": torch.uint8}
_TYPESTR = {"f64": "<f8", "f32": "<f4", "i64": "<i8", "i32": "<i4", "u8": "|u1", "bool": "|u1"}
_CTX = None


def listed():
    return [
        # One request of a service: thousands of rows, three statements, latency.
        {"name": "program_1k", "kind": "program", "n": 1000, "graph": False},
        # The README program at its own size.
        {"name": "program_1m", "kind": "program", "n": 1_000_000, "graph": False},
        # The largest sweep size, streaming reductions beyond L2.
        {"name": "reduce_f64_2p28", "kind": "reduce", "n": 1 << 28, "dtype": "f64", "values": "uniform", "offset": 0},
        # A ragged f32 column of measurements.
        {"name": "narrow_f32_20m", "kind": "narrow", "n": 20_000_003, "dtype": "f32"},
        # Half of the rows kept, the middle of the sweep's selectivities.
        {"name": "select_half_2p27", "kind": "select", "n": 1 << 27, "keep": 0.5, "offset": 0},
        # Uniform row numbers into a source far beyond L2.
        {"name": "gather_2p27", "kind": "gather", "n": 1 << 27, "m": 1 << 27, "dtype": "f64"},
        # Prefix sums over a column and over its segments (about 128 rows each).
        {"name": "scan_i64_2p27", "kind": "scan", "n": 1 << 27, "dtype": "i64", "segment": 128},
        # Float running sums in the language's own order, and per-bucket float sums.
        {"name": "fsum_33m", "kind": "fsum", "n": (1 << 25) + 13, "segment": 128, "buckets": 1024},
        # Keys over a full 32-bit range, as in the sort and group-by pipeline.
        {"name": "sort_u32_40m", "kind": "sort", "n": 40_000_011, "keys": "range32"},
        # A group-by with many rows and a moderate number of groups.
        {"name": "group_30m", "kind": "group", "n": 30_000_001, "distinct": 1 << 16, "dtype": "i64"},
        # Thousands of uneven arrays, one statement each.
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 10, "hi": 16},
        # Column arithmetic over three ragged columns.
        {"name": "expr_50m", "kind": "expr", "n": 50_000_017, "offset": 0},
    ]


def _log(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["program", "reduce", "narrow", "select", "gather", "scan", "fsum", "sort", "group", "batch",
                       "expr"])
    offset = rng.choice([0, 0, 0, 1])  # a slice of a longer column: rows off the 16-byte grid
    if kind == "program":
        return {"kind": kind, "n": _log(rng, 1000, 10_000_000), "graph": rng.random() < 0.25}
    if kind == "reduce":
        # Values around zero make the ordered sums hard: a smaller column.
        values = rng.choice(["uniform", "uniform", "normal"])
        return {"kind": kind, "n": _log(rng, 1 << 14, 1 << 22 if values == "normal" else (1 << 28) - 1), "dtype": rng.choice(["f64", "f64", "i64"]),
                "values": values, "offset": offset}
    if kind == "narrow":
        return {"kind": kind, "n": _log(rng, 1 << 14, 20_000_000), "dtype": rng.choice(["f32", "i32"])}
    if kind == "select":
        return {"kind": kind, "n": _log(rng, 1 << 14, 1 << 27), "keep": rng.choice([0.01, 0.5, 0.99]),
                "offset": offset}
    if kind == "gather":
        return {"kind": kind, "n": _log(rng, 1 << 14, 1 << 27), "m": _log(rng, 1 << 10, 1 << 27),
                "dtype": rng.choice(["f64", "i64", "i32"])}
    if kind == "scan":
        return {"kind": kind, "n": _log(rng, 1 << 14, 1 << 27), "dtype": rng.choice(["i64", "i64", "f64", "i32"]),
                "segment": _log(rng, 16, 1 << 14)}
    if kind == "fsum":
        return {"kind": kind, "n": _log(rng, 1 << 14, 1 << 25), "segment": _log(rng, 16, 1 << 14),
                "buckets": _log(rng, 64, 1 << 20)}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 1000, 40_000_000), "keys": rng.choice(["range32", "zipf", "i32"])}
    if kind == "group":
        n = _log(rng, 1 << 12, 30_000_000)
        return {"kind": kind, "n": n, "distinct": _log(rng, 10, n), "dtype": rng.choice(["i64", "i32"])}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 64, 4096), "lo": rng.randint(6, 10), "hi": rng.randint(12, 16)}
    return {"kind": kind, "n": _log(rng, 1 << 14, 50_000_000), "offset": offset}


# ---------------------------------------------------------------- inputs


def _context():
    """The program's one context, opened on its first use."""
    global _CTX
    if _CTX is None:
        _CTX = vk.Context()
    return _CTX


class _Rows:
    """Device rows of a framework array, for torch to read in place (it keeps the array alive)."""

    def __init__(self, array):
        self.array = array
        self.__cuda_array_interface__ = {"version": 3, "shape": (len(array),), "typestr": _TYPESTR[array.type],
                                         "data": (array.device_ptr or 0, False), "strides": None}


def _tensor(array):
    if len(array) == 0:
        return torch.empty(0, dtype=_TORCH[array.type], device=_DEVICE)
    return torch.as_tensor(_Rows(array), device=_DEVICE)


def _array(ctx, t, type_name, offset=0):
    """A framework array with the tensor's rows (`offset`: a slice that starts that many rows in)."""
    whole = ctx.new_array(type_name, t.numel() + offset)
    ctx.synchronize()
    _tensor(whole)[offset:].copy_(t)
    torch.cuda.synchronize()
    return whole.slice(offset, offset + t.numel()) if offset else whole


def _generator(seed):
    g = torch.Generator(device=_DEVICE)
    g.manual_seed(seed)
    return g


def _uniform(g, n, dtype=torch.float64):
    return torch.rand(n, generator=g, device=_DEVICE, dtype=dtype)


def _integers(g, lo, hi, n, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), generator=g, device=_DEVICE, dtype=dtype)


def _zipf(g, n):
    """64-bit keys of 2^20 distinct values whose frequencies follow Zipf's law (s = 1.1)."""
    w = torch.arange(1, (1 << 20) + 1, device=_DEVICE, dtype=torch.float64).pow(-1.1)
    cdf = torch.cumsum(w, 0)
    rank = torch.searchsorted(cdf, _uniform(g, n) * cdf[-1])
    return (rank + 1) * 0x1E3779B97F4A7C15


def _starts(g, n, segment):
    s = (_uniform(g, n, torch.float32) < 1.0 / segment).to(torch.uint8)
    s[0] = 1
    return s


def _lengths(case, seed):
    """The arrays' lengths, log-uniform: the same ones for every seed, in another order."""
    lens = [int(2 ** u) for u in np.random.default_rng(13).uniform(case["lo"], case["hi"], case["count"])]
    return np.random.default_rng(seed).permutation(lens).tolist()


def _chosen(g, n, keep):
    """A mask of exactly keep * n rows (at least one), anywhere."""
    r = _uniform(g, n)
    return r <= torch.kthvalue(r, max(1, int(keep * n))).values


def _around(chosen, u, limit):
    """Values in [0, 1) made from uniform u: above `limit` in the chosen rows, else at most `limit`."""
    low = torch.nextafter(torch.tensor(limit, dtype=u.dtype), torch.tensor(1.0, dtype=u.dtype)).item()
    return torch.where(chosen, (limit + (1.0 - limit) * u).clamp_min(low), limit * u)


def _inputs(case, seed):
    """The case's columns as torch tensors on the GPU, from the seed alone."""
    g, kind = _generator(seed), case["kind"]
    if kind == "program":
        return {"x": _uniform(g, case["n"]), "y": _uniform(g, case["n"])}
    n = case.get("n")
    if kind == "reduce":
        if case["dtype"] == "i64":
            return {"x": _integers(g, -1 << 40, 1 << 40, n), "y": _integers(g, -1 << 20, 1 << 20, n)}
        if case["values"] == "normal":
            return {"x": torch.randn(n, generator=g, device=_DEVICE, dtype=torch.float64),
                    "y": torch.randn(n, generator=g, device=_DEVICE, dtype=torch.float64)}
        return {"x": _uniform(g, n), "y": _uniform(g, n)}
    if kind == "narrow":
        kept = _chosen(g, n, 0.25)
        if case["dtype"] == "f32":
            return {"x": _around(kept, _uniform(g, n, torch.float32), 0.75), "y": _uniform(g, n, torch.float32)}
        high, low = _integers(g, (1 << 19) + 1, 1 << 20, n, torch.int32), _integers(g, -1 << 20, 1 << 19, n, torch.int32)
        return {"x": torch.where(kept, high, low), "y": _integers(g, -1 << 10, 1 << 10, n, torch.int32)}
    if kind == "select":
        return {"x": _around(_chosen(g, n, case["keep"]), _uniform(g, n), 1.0 - case["keep"]),
                "v": _integers(g, -1 << 40, 1 << 40, n), "m": _chosen(g, n, case["keep"]).to(torch.uint8)}
    if kind == "gather":
        m = case["m"]
        src = _uniform(g, m) if case["dtype"] == "f64" else _integers(g, -1 << 30, 1 << 30, m, _TORCH[case["dtype"]])
        return {"x": src, "i": _integers(g, 0, m, n)}
    if kind == "scan":
        if case["dtype"] == "f64":
            x = torch.randn(n, generator=g, device=_DEVICE, dtype=torch.float64)
        else:
            x = _integers(g, -1 << 20, 1 << 20, n, _TORCH[case["dtype"]])
        return {"x": x, "s": _starts(g, n, case["segment"])}
    if kind == "fsum":
        return {"x": _uniform(g, n), "s": _starts(g, n, case["segment"]), "k": _integers(g, 0, case["buckets"], n)}
    if kind == "sort":
        if case["keys"] == "zipf":
            k = _zipf(g, n)
        elif case["keys"] == "i32":
            k = _integers(g, -1 << 31, 1 << 31, n).to(torch.int32)
        else:
            k = _integers(g, 0, 1 << 32, n)
        return {"k": k, "v": _uniform(g, n)}
    if kind == "group":
        d = case["distinct"]
        k = _integers(g, 0, d, n)
        k[torch.arange(d, device=_DEVICE) * n // d] = torch.randperm(d, generator=g, device=_DEVICE)  # each occurs
        k *= 0x1E3779B97F4A7C15  # identifiers, not small numbers
        return {"k": k, "v": _integers(g, -1 << 20, 1 << 20, n, _TORCH[case["dtype"]])}
    if kind == "batch":
        rows = sum(_lengths(case, seed))
        return {"x": _uniform(g, rows), "k": _integers(g, 0, 1 << 16, rows)}
    return {"x": _uniform(g, n), "y": _uniform(g, n), "z": _uniform(g, n)}


_TYPES = {"program": {"x": "f64", "y": "f64"}, "select": {"x": "f64", "v": "i64", "m": "bool"},
          "fsum": {"x": "f64", "s": "bool", "k": "i64"}, "batch": {"x": "f64", "k": "i64"},
          "expr": {"x": "f64", "y": "f64", "z": "f64"}}


def _types(case):
    kind, d = case["kind"], case.get("dtype")
    if kind in ("reduce", "narrow"):
        return {"x": d, "y": d}
    if kind == "gather":
        return {"x": d, "i": "i64"}
    if kind == "scan":
        return {"x": d, "s": "bool"}
    if kind == "sort":
        return {"k": "i32" if case["keys"] == "i32" else "i64", "v": "f64"}
    if kind == "group":
        return {"k": "i64", "v": d}
    return _TYPES[kind]


def prepare(case, seed):
    ctx = _context()
    types = _types(case)
    s = {k: _array(ctx, t, types[k], case.get("offset", 0)) for k, t in _inputs(case, seed).items()}
    if case["kind"] == "batch":
        s = _prepare_batch(ctx, case, seed, s)
    elif case["kind"] == "program" and case["graph"]:
        s = _prepare_graph(ctx, s)
    return dict(s, case=case, ctx=ctx)


def _prepare_batch(ctx, case, seed, s):
    """The arrays are views of two long columns, and their orders go to views of one column."""
    ends = np.concatenate([[0], np.cumsum(_lengths(case, seed))]).tolist()
    spans = list(zip(ends[:-1], ends[1:]))
    order = ctx.new_array("i64", ends[-1])
    count = case["count"]
    return {"order": order, "sums": ctx.new_array("f64", count), "counts": ctx.new_array("i64", count),
            "xs": ctx.batch([s["x"].slice(a, b) for a, b in spans]),
            "ks": ctx.batch([s["k"].slice(a, b) for a, b in spans]),
            "orders": ctx.batch([order.slice(a, b) for a, b in spans])}


def _prepare_graph(ctx, s):
    """The program's statements with their results left on the device, captured once."""
    fs, ints = ctx.new_array("f64", 1), ctx.new_array("i64", 2)

    def statements():
        ctx.call_into("dot_f64", s["x"], s["y"], out=fs, row=0)
        ctx.call_into("count_gt_f64", s["x"], 0.5, out=ints, row=0)
        ctx.call_into("count_gt_f64", s["x"], 0.99, out=ints, row=1)

    statements()
    ctx.synchronize()
    ctx.graph_begin()
    statements()
    return dict(s, graph=ctx.graph_end(), floats=fs, ints=ints)


# ---------------------------------------------------------------- one pass


def run(state):
    return _RUN[state["case"]["kind"]](state["ctx"], state["case"], state)


def _run_program(ctx, case, s):
    if case["graph"]:
        s["graph"].launch()
        return [_tensor(s["floats"]), _tensor(s["ints"])]
    kept = ctx.call("filter_gt_f64", s["x"], 0.99)
    return [ctx.call("dot_f64", s["x"], s["y"]), ctx.call("count_gt_f64", s["x"], 0.5), ctx.call("length_f64", kept)]


def _run_reduce(ctx, case, s):
    d, x = case["dtype"], s["x"]
    limit = 0.25 if d == "f64" else 1 << 30
    return [ctx.call("reduce_add_" + d, x), ctx.call("dot_" + d, x, s["y"]), ctx.call("reduce_min_" + d, x),
            ctx.call("reduce_max_" + d, x), ctx.call("argmin_" + d, x), ctx.call("argmax_" + d, x),
            ctx.call("count_lt_" + d, x, limit)]


def _run_narrow(ctx, case, s):
    d, x = case["dtype"], s["x"]
    limit = vk.Scalar("f32", 0.75) if d == "f32" else vk.Scalar("i32", 1 << 19)
    return [ctx.call("reduce_add_" + d, x), ctx.call("dot_" + d, x, s["y"]), ctx.call("reduce_max_" + d, x),
            ctx.call("argmin_" + d, x), ctx.call("count_gt_" + d, x, limit),
            _tensor(ctx.call("filter_gt_" + d, x, limit))]


def _run_select(ctx, case, s):
    return [_tensor(ctx.call("filter_gt_f64", s["x"], 1.0 - case["keep"])),
            _tensor(ctx.call("compress_i64", s["v"], s["m"])), _tensor(ctx.call("where", s["m"]))]


def _run_gather(ctx, case, s):
    return [_tensor(ctx.call("gather_" + case["dtype"], s["x"], s["i"]))]


def _run_scan(ctx, case, s):
    op = "max_f64" if case["dtype"] == "f64" else "add_" + case["dtype"]
    return [_tensor(ctx.call("scan_" + op, s["x"])), _tensor(ctx.call("scan_by_" + op, s["x"], s["s"]))]


def _run_fsum(ctx, case, s):
    return [_tensor(ctx.call("scan_add_f64", s["x"])), _tensor(ctx.call("scan_by_add_f64", s["x"], s["s"])),
            _tensor(ctx.call("reduce_into_add_f64", s["k"], s["x"], case["buckets"]))]


def _run_sort(ctx, case, s):
    order = ctx.call("argsort_i32" if case["keys"] == "i32" else "argsort_i64", s["k"])
    return [_tensor(order), _tensor(ctx.call("gather_f64", s["v"], order))]


def _run_group(ctx, case, s):
    ids = ctx.call("group_id_i64", s["k"])
    groups = ctx.call("reduce_max_i64", ids) + 1
    return [_tensor(ids), groups, _tensor(ctx.call("reduce_into_add_" + case["dtype"], ids, s["v"], groups)),
            _tensor(ctx.call("histogram", ids, groups))]


def _run_batch(ctx, case, s):
    ctx.batch_filter_sum(s["xs"], "gt", 0.9, s["sums"])
    ctx.batch_count(s["xs"], "lt", 0.5, s["counts"])
    ctx.batch_argsort(s["ks"], s["orders"], 0b11)  # keys below 2^16: two bytes vary
    return [_tensor(s["sums"]), _tensor(s["counts"]), _tensor(s["order"])]


def _run_expr(ctx, case, s):
    xyz, k = [s["x"], s["y"], s["z"]], vk.region_kernel
    return [_tensor(ctx.region([("mul_f64", (0, 1)), ("add_f64", (k(0), 2))], xyz)),
            ctx.region_reduce("count", [k(1)], [("mul_f64", (0, 1)), ("gt_f64", (k(0), 2))], [s["x"], s["y"], 0.25]),
            ctx.region_reduce("reduce_min_f64", [k(1)], [("mul_f64", (0, 1)), ("add_f64", (k(0), 2))], xyz)]


_RUN = {"program": _run_program, "reduce": _run_reduce, "narrow": _run_narrow, "select": _run_select,
        "gather": _run_gather, "scan": _run_scan, "fsum": _run_fsum, "sort": _run_sort, "group": _run_group,
        "batch": _run_batch, "expr": _run_expr}


# ---------------------------------------------------------------- exact results and work


def exact(case, seed):
    """The float results in 64 bits (whole numbers are None: they are compared bit for bit)."""
    t, kind = _inputs(case, seed), case["kind"]
    if kind == "program":
        dot = (t["x"] * t["y"]).sum()
        return [dot.reshape(1), None] if case["graph"] else [float(dot), None, None]
    if kind == "reduce":
        if case["dtype"] != "f64":
            return None
        x, y = t["x"], t["y"]
        return [float(x.sum()), float((x * y).sum()), float(x.min()), float(x.max()), None, None, None]
    if kind == "narrow":
        if case["dtype"] != "f32":
            return None
        x, y = t["x"].double(), t["y"].double()
        return [float(x.sum()), float((x * y).sum()), float(x.max()), None, None, x[t["x"] > 0.75]]
    if kind == "select":
        return [t["x"][t["x"] > 1.0 - case["keep"]], None, None]
    if kind == "gather":
        return [t["x"][t["i"]]] if case["dtype"] == "f64" else None
    if kind == "scan":
        return [torch.cummax(t["x"], 0).values, None] if case["dtype"] == "f64" else None
    if kind == "fsum":
        run_sum = torch.cumsum(t["x"], 0)
        number = torch.cumsum(t["s"], 0, dtype=torch.int64) - 1  # the row's segment
        first = t["s"].nonzero().squeeze(1)
        before = torch.where(first > 0, run_sum[first - 1], torch.zeros_like(run_sum[first]))
        sums = torch.zeros(case["buckets"], dtype=torch.float64, device=_DEVICE).index_add_(0, t["k"], t["x"])
        return [run_sum, run_sum - before[number], sums]
    if kind == "sort":
        return [None, t["v"][torch.argsort(t["k"], stable=True)]]
    if kind == "batch":
        lens = torch.tensor(_lengths(case, seed), device=_DEVICE)
        number = torch.repeat_interleave(torch.arange(case["count"], device=_DEVICE), lens)
        kept = torch.where(t["x"] > 0.9, t["x"], torch.zeros_like(t["x"]))
        return [torch.zeros(case["count"], dtype=torch.float64, device=_DEVICE).index_add_(0, number, kept), None, None]
    if kind == "expr":
        v = t["x"] * t["y"] + t["z"]
        return [v, None, float(v.min())]
    return None


def work(case):
    """Bytes: each call's inputs read once and its results written once. Operations: the adds and products."""
    kind, n = case["kind"], case.get("n", 0)
    w = {"f64": 8, "i64": 8, "f32": 4, "i32": 4}.get(case.get("dtype"), 8)
    if kind == "program":
        return {"bytes": (16 + 8 + 8) * n + (0 if case["graph"] else 0.08 * n), "flops": 2 * n}
    if kind == "reduce":
        return {"bytes": 8 * w * n, "flops": 3 * n}
    if kind == "narrow":
        return {"bytes": (7 * w + (w + 1) * 0.25) * n, "flops": 3 * n}
    if kind == "select":
        return {"bytes": (8 + 9 + 1 + 24 * case["keep"]) * n, "flops": 0}
    if kind == "gather":
        return {"bytes": (8 + w) * n + w * min(n, case["m"]), "flops": 0}
    if kind == "scan":
        out = 8 if case["dtype"] == "i32" else w
        return {"bytes": (2 * w + 2 * out + 1) * n, "flops": 0}
    if kind == "fsum":
        return {"bytes": (16 + 17 + 16) * n + 8 * case["buckets"], "flops": 3 * n}
    if kind == "sort":
        key = 4 if case["keys"] == "i32" else 8
        return {"bytes": (key + 8 + 24) * n, "flops": 0}
    if kind == "group":
        return {"bytes": (16 + 8 + 8 + w + 8) * n + 16 * min(n, case["distinct"]), "flops": 0}
    if kind == "batch":
        rows = case["count"] * (2.0 ** case["hi"] - 2.0 ** case["lo"]) / ((case["hi"] - case["lo"]) * math.log(2))
        return {"bytes": 32 * rows, "flops": 0.1 * rows}
    return {"bytes": (32 + 16 + 24) * n, "flops": 5 * n}
