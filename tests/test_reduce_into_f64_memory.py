"""reduce_into_add_f64 where the sorted path's scratch cannot be allocated (k_reduce_into_f64.cu): the chains
are found by a scan, whose scratch does not grow with the buckets."""

import numpy as np
import pytest

import oracle
from helpers import varied

pytestmark = pytest.mark.gpu


def test_scratch_that_cannot_be_allocated():
    import verkehrt_gb300 as vk

    c = vk.Context(0)
    try:
        n, nb = 100_003, 50_000
        keys = (oracle.rand_i64(n, 3).view(np.uint64) % np.uint64(nb)).astype(np.int64)
        x = varied(n, 4)
        dk, dx = c.upload(keys), c.upload(x)
        want = oracle.reduce_into_add_f64(keys, x, nb).view(np.uint64)
        for at in range(1, 9):  # after the result: images, values, tables, and the chains' table last
            c.tune_set("fail_alloc_after", 0, at)
            got = c.call("reduce_into_add_f64", dk, dx, nb).numpy()
            assert c.tune_get("fail_alloc_after", 0) == -1, at
            assert np.array_equal(got.view(np.uint64), want), at
        keys[70_000] = nb
        dk = c.upload(keys)
        c.tune_set("fail_alloc_after", 0, 8)
        with pytest.raises(vk.KernelError, match="^bucket key %d out of range for %d buckets$" % (nb, nb)):
            c.call("reduce_into_add_f64", dk, dx, nb)
    finally:
        c.close()
