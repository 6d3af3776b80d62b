"""Folded regions of one f64 array at the turn between their two evaluators (k_elementwise.cu, folds_as_words)
and of four arrays: the bits of whole evaluation, with NaNs, signed zeros and rows off the 16-byte grid."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TURN = 1 << 22


def whole(ctx, kernels, inputs):
    values = []
    for name, args in kernels:
        values.append(ctx.call(name, *[inputs[a] if a >= 0 else values[-1 - a] for a in args]))
    return values[-1]


@pytest.mark.parametrize("n", [TURN - 1, TURN, TURN + 513])
@pytest.mark.parametrize("special", [False, True])
def test_one_array(ctx, n, special):
    import verkehrt_gb300 as vk

    k = vk.region_kernel
    x = oracle.rand_f64(n + 1, 3) - 0.5
    if special:
        x[n // 3] = np.nan
        x[n // 5] = -0.0
    for dx in (ctx.upload(x[:n]), ctx.upload(x).slice(1, n + 1)):
        for kernels in ([("mul_f64", (0, 1)), ("add_f64", (k(0), 0))], [("mul_f64", (0, 1)), ("neg_f64", (k(0),))],
                        [("abs_f64", (0,)), ("sqrt_f64", (k(0),)), ("div_f64", (k(1), 1))],
                        [("mul_f64", (0, 1)), ("abs_f64", (k(0),))],
                        [("mul_f64", (0, 0)), ("sub_f64", (k(0), 1)), ("max_f64", (k(1), 0))]):
            inputs = [dx, 0.375]
            want = whole(ctx, kernels, inputs)
            for root in ("reduce_min_f64", "reduce_max_f64", "argmin_f64", "argmax_f64"):
                got = ctx.region_reduce(root, [k(len(kernels) - 1)], kernels, inputs, raw=True)
                assert got[2] == ctx.call(root, want, raw=True)[2], (kernels, root)


def test_two_and_three_arrays(ctx):
    import verkehrt_gb300 as vk

    k = vk.region_kernel
    n = TURN + 77
    columns = [ctx.upload(oracle.rand_f64(n, s) - 0.5) for s in range(3)]
    for inputs in (columns[:2], columns):
        last = len(inputs) - 1
        for count in (2, 3, 5):
            kernels = [("mul_f64", (0, 1)), ("sub_f64", (k(0), last)), ("mul_f64", (k(1), 0)), ("neg_f64", (k(2),)),
                       ("add_f64", (k(3), last))][:count]
            want = whole(ctx, kernels, inputs)
            for root in ("reduce_max_f64", "argmin_f64"):
                got = ctx.region_reduce(root, [k(count - 1)], kernels, inputs, raw=True)
                assert got[2] == ctx.call(root, want, raw=True)[2], (count, root)


def test_negation(ctx):
    import verkehrt_gb300 as vk

    k = vk.region_kernel
    x = np.concatenate([oracle.rand_f64(5000, 1) - 0.5, [0.0, -0.0, np.inf, -np.inf, 5e-324, -5e-324]])
    dx = ctx.upload(x)
    got = ctx.region([("neg_f64", (0,)), ("neg_f64", (k(0),)), ("neg_f64", (k(1),))], [dx]).numpy()
    assert np.array_equal(got.view(np.uint64), (-x).view(np.uint64))
    assert ctx.region_reduce("count", [k(1)], [("neg_f64", (0,)), ("gt_f64", (k(0), 0))], [dx]) == int((-x > x).sum())


def test_four_arrays(ctx):
    import verkehrt_gb300 as vk

    k = vk.region_kernel
    for n in (1, 511, 512, 513, 1_000_003):
        inputs = [ctx.upload(oracle.rand_f64(n, s) - 0.5) for s in range(4)]
        kernels = [("mul_f64", (0, 1)), ("add_f64", (k(0), 2)), ("gt_f64", (k(1), 3)), ("select_f64", (k(2), k(1), k(0)))]
        want = whole(ctx, kernels, inputs)
        for root in ("reduce_min_f64", "argmax_f64"):
            got = ctx.region_reduce(root, [k(3)], kernels, inputs, raw=True)
            assert got[2] == ctx.call(root, want, raw=True)[2], (n, root)
