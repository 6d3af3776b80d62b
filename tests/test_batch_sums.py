"""Batched filtered sums (k_batch.cu) where a chunk of 2048 rows leaves survivors over for the next: arrays around
the chunk's size, none, few, most and all rows kept, specials among them; bit for bit against the oracle."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LENS = [0, 1, 15, 16, 17, 2047, 2048, 2049, 4096 + 15, 10_000, 65_536]


@pytest.mark.parametrize("limit", [-1.0, 0.003, 0.5, 0.97, 2.0])
def test_filter_sums(ctx, limit):
    x = oracle.rand_f64(sum(LENS), 11)
    x[5::1001] = 1e-310
    x[7::977] = -0.0
    dx = ctx.upload(x)
    ends = np.concatenate([[0], np.cumsum(LENS)])
    spans = [(int(a), int(b)) for a, b in zip(ends[:-1], ends[1:])]
    batch = ctx.batch([dx.slice(a, b) for a, b in spans])
    for cmp in ("lt", "gt"):
        sums = ctx.new_array("f64", len(LENS))
        ctx.batch_filter_sum(batch, cmp, limit, sums)
        for (a, b), got in zip(spans, sums.numpy()):
            part = x[a:b]
            kept = part[part < limit] if cmp == "lt" else part[part > limit]
            assert np.float64(got).tobytes() == np.float64(oracle.reduce_add_f64(kept)).tobytes(), (cmp, a, b)
