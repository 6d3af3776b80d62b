"""reduce_into_add_f64 at the turns of its dispatch (k_reduce_into_f64.cu): masked sums, sorted chains
staged or read by their threads, one to four radix passes, and chains found by a scan; bit for bit
against the oracle, and the first bad key wherever it lies."""

import numpy as np
import pytest

import oracle
from helpers import varied

pytestmark = pytest.mark.gpu


def bits(v):
    return np.asarray(v, dtype=np.float64).view(np.uint64)


@pytest.mark.parametrize("nb", [1, 2, 16, 17, 256, 4096, 70_000, 1 << 20, (1 << 24) + 1])
def test_paths_equal_the_oracle(ctx, nb):
    for n in (16, 4099, 65_551, 1_000_003):
        x = varied(n, n)
        u = oracle.rand_i64(n, nb).view(np.uint64)
        for keys in ((u % np.uint64(nb)).astype(np.int64), (u % np.uint64(max(1, nb // 3))).astype(np.int64) // 7):
            got = ctx.call("reduce_into_add_f64", ctx.upload(keys), ctx.upload(x), nb).numpy()
            assert np.array_equal(bits(got), bits(oracle.reduce_into_add_f64(keys, x, nb))), (n, nb)


def test_bad_keys_in_the_blocks_and_in_the_tail(ctx):
    n, nb = 100_003, 64
    x = ctx.upload(varied(n, 1))
    for at, bad in ((70, -3), (n - 1, 64), (n - 2, 1 << 40), (0, -2**63)):
        keys = (oracle.rand_i64(n, 3).view(np.uint64) % np.uint64(nb)).astype(np.int64)
        keys[at] = bad
        with pytest.raises(Exception, match="^bucket key %d out of range for %d buckets$" % (bad, nb)):
            ctx.call("reduce_into_add_f64", ctx.upload(keys), x, nb)
    assert len(ctx.call("reduce_into_add_f64", ctx.upload(keys % nb), x, nb)) == nb
