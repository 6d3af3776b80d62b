"""The f64 region evaluator (k_elementwise.cu) at the edges of its steps (1024 rows of one or two
arrays, 512 of three or four), on slices off the 16-byte grid, storing, counting and folding, with
comparisons against constants on either side; against the kernels run one by one."""

import numpy as np
import pytest

import oracle
from helpers import with_specials
from verkehrt_gb300 import region_kernel as k

pytestmark = pytest.mark.gpu


def bits(v):
    return np.asarray(v, dtype=np.float64).view(np.uint64)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 1023, 1024, 1025, 70_001])
def test_f64_regions_equal_whole_evaluation(ctx, n, off):
    c = ctx.call
    cols = [with_specials(n + off, 3 + i) for i in range(4)]
    x, y, z, w = (ctx.upload(v).slice(off, n + off) for v in cols)
    clean = ctx.upload(oracle.rand_f64(n + off, 5) - 0.5).slice(off, n + off)
    for cmp in ("lt", "le", "gt", "ge", "eq", "ne"):
        for const in (0.0, -0.0, 0.25, np.inf, np.nan):
            for args, whole in (((k(0), 1), lambda: c(cmp + "_f64", c("neg_f64", x), const)),
                                ((1, k(0)), lambda: c(cmp + "_f64", const, c("neg_f64", x)))):
                ks = [("neg_f64", (0,)), (cmp + "_f64", args)]
                assert np.array_equal(ctx.region(ks, [x, const]).numpy(), whole().numpy()), (cmp, const)
                assert ctx.region_reduce("count", [k(1)], ks, [x, const]) == c("count", whole()), (cmp, const)
        ks = [("mul_f64", (0, 1)), (cmp + "_f64", (k(0), 2)), ("select_f64", (k(1), 3, k(0)))]
        want = c("select_f64", c(cmp + "_f64", c("mul_f64", x, y), z), w, c("mul_f64", x, y))
        got = ctx.region(ks, [x, y, z, w]).numpy()
        nan = np.isnan(want.numpy())
        assert np.array_equal(np.isnan(got), nan) and np.array_equal(bits(got[~nan]), bits(want.numpy()[~nan])), cmp
    for a, b in ((x, y), (clean, clean), (clean, x)):
        for root in ("reduce_min_f64", "reduce_max_f64", "argmin_f64", "argmax_f64"):
            for ks, whole in (([("mul_f64", (0, 1))], lambda: c("mul_f64", a, b)),
                              ([("add_f64", (0, 1)), ("mul_f64", (k(0), 2))], lambda: c("mul_f64", c("add_f64", a, b), clean))):
                got = ctx.region_reduce(root, [k(len(ks) - 1)], ks, [a, b, clean][:len(ks) + 1], raw=True)
                want = c(root, whole(), raw=True)
                assert got[2] == want[2] or (np.isnan(got[1]) and np.isnan(want[1])), (root, got, want)
