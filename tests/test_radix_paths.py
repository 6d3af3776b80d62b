"""The radix passes of argsort and the batched argsort where their dispatch turns (k_sort.cu, k_batch.cu):
images of the varying bytes or of the distance from the least key, 32 or 64 bits wide, one to eight
passes; batched images in 32 bits, in 64 bits, and too wide for one. Whole numbers, bit for bit."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def keys(kind, n, seed):
    r = oracle.rand_i64(n, seed)
    u = r.view(np.uint64)
    return {
        "signed_small": (u % np.uint64(1000)).astype(np.int64) - 500,       # every byte varies, the range does not
        "signed_33bit": (u % np.uint64(1 << 33)).astype(np.int64) - (1 << 32),
        "high_bytes": ((u & np.uint64(0xFFFF)) << np.uint64(48)).view(np.int64),  # two bytes vary, a wide range
        "offset_range": (u % np.uint64(70_000)).astype(np.int64) + (0xFFFFFF00 - 5),  # crosses 2^32
        "one_pass": (u % np.uint64(256)).astype(np.int64) - 128,
        "constant": np.full(n, -7, dtype=np.int64),
        "all": r,
    }[kind]


@pytest.mark.parametrize("kind", ["signed_small", "signed_33bit", "high_bytes", "offset_range", "one_pass", "constant", "all"])
def test_argsort_images(ctx, kind):
    for n in (8193, 2 * 2048 * 7, 2 * 3072 * 5 + 1, 4096 * 9 - 1, 1_200_001):
        k = keys(kind, n, n)
        assert np.array_equal(ctx.call("argsort_i64", ctx.upload(k)).numpy(), oracle.argsort_i64(k)), n
        i32 = k.astype(np.int32)
        assert np.array_equal(ctx.call("argsort_i32", ctx.upload(i32)).numpy(), oracle.argsort_i64(i32.astype(np.int64))), n
        u8 = k.astype(np.uint8)
        assert np.array_equal(ctx.call("argsort_u8", ctx.upload(u8)).numpy(), oracle.argsort_i64(u8.astype(np.int64))), n
        u64 = k.view(np.uint64)
        assert np.array_equal(ctx.call("argsort_u64", ctx.upload(u64)).numpy(),
                              oracle.argsort_i64((u64 ^ np.uint64(1 << 63)).view(np.int64))), n
        # A slice off the 16-byte grid.
        assert np.array_equal(ctx.call("argsort_i64", ctx.upload(k).slice(1, n)).numpy(), oracle.argsort_i64(k[1:])), n


@pytest.mark.parametrize("arrays", [1, 256, 300])
@pytest.mark.parametrize("digits", [0b1, 0b11, 0b111, 0b10010001, 0b111111, 0b1111111, 0])
def test_batched_argsort_images(ctx, arrays, digits):
    rng = np.random.default_rng(arrays)
    lens = rng.integers(0, 700, arrays)
    lens[0] = 9001
    mask = sum(0xFF << (8 * k) for k in range(8) if (digits or 0xFF) >> k & 1)
    ks = [((oracle.rand_i64(int(n), 90 + i).view(np.uint64) & np.uint64(mask)) ^ np.uint64(1 << 63)).view(np.int64)
          for i, n in enumerate(lens)]
    outs = [ctx.new_array("i64", int(n)) for n in lens]
    ctx.batch_argsort(ctx.batch([ctx.upload(k) for k in ks]), ctx.batch(outs), digits)
    for k, o in zip(ks, outs):
        assert np.array_equal(o.numpy(), oracle.argsort_i64(k)), len(k)
