"""Scans of every word width (fold_scan.cuh) at the edges of lanes, steps, slices and tiles, on rows off the
vector grid, with starts nowhere, everywhere and at those edges, and with NaNs (a segment's first row keeps
its payload), infinities and signed zeros; bit for bit against the oracle."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

CASES = [("i64", "add"), ("u64", "mul"), ("i64", "min"), ("u64", "max"), ("f64", "min"), ("f64", "max"), ("f32", "min"),
         ("f32", "max"), ("i32", "add"), ("i32", "max"), ("i32", "mul"), ("u8", "add"), ("u8", "mul"), ("u8", "xor"),
         ("bool", "and"), ("bool", "xor")]
DT = {"i64": np.int64, "u64": np.uint64, "f64": np.float64, "f32": np.float32, "i32": np.int32, "u8": np.uint8,
      "bool": np.bool_}


def rows(t, n, seed):
    u = oracle.rand_i64(n, seed).view(np.uint64)
    if t == "bool":
        return (u % np.uint64(9) != 0).astype(np.bool_)
    if t not in ("f64", "f32"):
        return u.astype(DT[t])
    x = (u.view(np.int64) >> 40).astype(DT[t])
    bits = x.view(np.uint64 if t == "f64" else np.uint32)
    pick = (u % np.uint64(97)).astype(np.int64)
    specials = ([0x7ff8000000000000, 0xfff8000000000123, 0x7ff0000000000001, 0x7ff0000000000000, 0xfff0000000000000,
                 0x8000000000000000, 0] if t == "f64" else
                [0x7fc00000, 0xffc00123, 0x7f800001, 0x7f800000, 0xff800000, 0x80000000, 0])
    for i, b in enumerate(specials):
        bits[(pick == i) & (np.arange(n) % (1 + 40 * (i < 3)) == 0)] = b
    return x


def starts(kind, n, seed):
    s = np.zeros(n, dtype=np.bool_)
    i = np.arange(n)
    if kind == "all":
        s[:] = True
    elif kind == "edges":
        s[(i % 8192 == 0) | (i % 512 == 511) | (i % 1024 == 0) | (i % 128 == 4)] = True
    elif kind == "few":
        s[oracle.rand_i64(n, seed).view(np.uint64) % np.uint64(700) == 0] = True
    return s


def bits(a):
    return np.ascontiguousarray(a).view(np.uint8)


@pytest.mark.parametrize("t,f", CASES)
def test_scan_folds(ctx, t, f):
    for n in (1, 3, 128, 513, 8191, 8192, 8193, 16_383, 16_385, 70_001):
        for off in (0, 1):
            x = rows(t, n, n)
            whole = np.concatenate([x[:off], x])
            dx = ctx.upload(whole).slice(off, off + n)
            assert np.array_equal(bits(ctx.call("scan_%s_%s" % (f, t), dx).numpy()), bits(oracle.scan(t, f, x))), (n, off)
            for kind in ("none", "all", "edges", "few"):
                s = starts(kind, n, 7)
                ds = ctx.upload(np.concatenate([s[:off], s])).slice(off, off + n)
                got = ctx.call("scan_by_%s_%s" % (f, t), dx, ds).numpy()
                want = oracle.scan(t, f, x, s)
                if t in ("f64", "f32"):
                    want = want.copy()
                    first = s & np.isnan(x)
                    want[first] = x[first]
                assert np.array_equal(bits(got), bits(want)), (n, off, kind)
