"""Batched argsort with each array sorted for itself (radix.h, radix_segs): arrays around the tiles' sizes,
empty ones among them, off the 16-byte grid, keys with many equal ones, digits side by side and apart, one to
eight of them; against the oracle's argsort of each array's chosen digits."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LENS = [3072, 1, 0, 3071, 3073, 6144, 20_001, 2048, 0, 12_288, 33_333, 2047, 2049, 5]


@pytest.mark.parametrize("digits", [0, 0b1, 0b11, 0b110, 0b101, 0b1111, 0b10110011, 0b10000000])
@pytest.mark.parametrize("count", [1, len(LENS), 300, 301])
def test_argsort(ctx, digits, count):
    lens = [20_001] if count == 1 else (LENS if count == len(LENS) else (LENS * 24)[:300] if count == 300 else [2048, 1025, 1999] * 100 + [2049])
    off = 1
    k = oracle.rand_i64(off + sum(lens), 7)
    k[k % 3 == 0] &= 0x0301  # many equal keys
    dk, do = ctx.upload(k), ctx.new_array("i64", off + sum(lens))
    ends = off + np.concatenate([[0], np.cumsum(lens)])
    spans = [(int(a), int(b)) for a, b in zip(ends[:-1], ends[1:])]
    keys, outs = ctx.batch([dk.slice(a, b) for a, b in spans]), ctx.batch([do.slice(a, b) for a, b in spans])
    for _ in range(2):
        ctx.batch_argsort(keys, outs, digits)
    got = do.numpy()
    mask = sum(0xff << (8 * d) for d in range(8) if (digits or 0xff) >> d & 1)
    image = (k.view(np.uint64) ^ np.uint64(1 << 63)) & np.uint64(mask)
    for a, b in spans:
        assert np.array_equal(got[a:b], np.argsort(image[a:b], kind="stable")), (a, b)
