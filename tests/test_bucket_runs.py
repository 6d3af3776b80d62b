"""Bucket counts and sums over keys in runs (k_index.cu): runs that fill groups of 32 rows, end inside them and
go on over them, few and many keys, keys that differ in their high halves alone, values over the whole 64 bits,
the last group short, and a bad key inside a run."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 2, 4, 31, 32, 33, 64, 1000, 100_000])
@pytest.mark.parametrize("nb", [1, 3, 5000, 300_000])
def test_runs(ctx, length, nb):
    for n in (1, 31, 32, 33, 255, 257, 100_003):
        k = np.repeat(oracle.rand_i64(n // length + 1, 7) % nb, length)[:n].astype(np.int64)
        v = oracle.rand_i64(n, 9)
        want = np.zeros(nb, np.int64)
        np.add.at(want, k, v)
        for keys in (k, np.sort(k)):
            dk = ctx.upload(keys)
            assert np.array_equal(ctx.call("histogram", dk, nb).numpy(), np.bincount(k, minlength=nb)), n
        assert np.array_equal(ctx.call("reduce_into_add_i64", ctx.upload(k), ctx.upload(v), nb).numpy(), want), n


def test_a_bad_key_inside_a_run(ctx):
    n = 10_000
    for at, bad in ((500, -1), (9_999, 7), (0, 1 << 40), (4_000, (1 << 33) + 2)):  # the last: another key's low half
        k = np.repeat(np.arange(5), 2000)
        k[at] = bad
        for call in (("histogram", ctx.upload(k), 7), ("reduce_into_add_i64", ctx.upload(k), ctx.upload(k), 7)):
            with pytest.raises(Exception, match="^bucket key %d out of range for 7 buckets$" % bad):
                ctx.call(*call)


def test_runs_of_keys_with_one_low_half(ctx):
    k = np.repeat(np.array([1, (1 << 32) + 1, 1, (2 << 32) + 1]), [40, 32, 5, 51])
    with pytest.raises(Exception, match="^bucket key 4294967297 out of range for 7 buckets$"):
        ctx.call("histogram", ctx.upload(k), 7)
