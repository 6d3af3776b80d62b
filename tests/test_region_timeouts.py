"""A folded region reports a wait that ran out in work enqueued before it (k_region.cu), as every call does that
waits for the device: a scan whose lookback polls for records that no block writes, with each wait bounded to
a few dozen polls (the hooks of tests/test_failure_paths.py)."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def test_folds_report_an_earlier_timeout():
    import verkehrt_gb300 as vk

    c = vk.Context(0)
    try:
        n = 1 << 22
        dv = c.upload(oracle.rand_i64(n, 3) >> 20)
        x = oracle.rand_f64(5000, 4)
        dx = c.upload(x)
        k = vk.region_kernel
        folds = [("reduce_min_f64", [("mul_f64", (0, 0)), ("add_f64", (k(0), 0))], [dx], float((x * x + x).min())),
                 ("argmax_f64", [("mul_f64", (0, 0)), ("add_f64", (k(0), 0))], [dx], int((x * x + x).argmax())),
                 ("reduce_max_i64", [("add_i64", (0, 0)), ("sub_i64", (k(0), 0))], [dv], int((oracle.rand_i64(n, 3) >> 20).max()))]
        c.call("scan_add_i64", dv).numpy()
        for root, kernels, inputs, want in folds:
            c.tune_set("spin_limit", 0, 64)
            c.tune_set("lookback_never_ready", 0, 1)
            c.call("scan_add_i64", dv)
            with pytest.raises(vk.KernelError) as e:
                c.region_reduce(root, [k(1)], kernels, inputs)
            assert (e.value.status, e.value.message) == ("TIMEOUT", "a device-side wait gave up")
            c.tune_set("lookback_never_ready", 0, 0)
            c.tune_set("spin_limit", 0, 0)
            assert c.region_reduce(root, [k(1)], kernels, inputs) == want
    finally:
        c.close()
