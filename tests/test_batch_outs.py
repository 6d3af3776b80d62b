"""Batched argsort into one batch of outputs after another (k_batch.cu): output batches that are freed
between calls, others of more sets than the tables kept, captured ones replayed among them, and a call whose
scratch could not be allocated."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LONG, SHORT = [5000, 3072, 1, 7000, 0, 2048], [40, 7, 100, 0, 33, 256]  # sorted for themselves, and together


def column(lens, seed):
    k = oracle.rand_i64(sum(lens), seed) % 1000
    ends = np.concatenate([[0], np.cumsum(lens)]).tolist()
    return k, list(zip(ends[:-1], ends[1:]))


def check(order, k, spans):
    got = order.numpy()
    for a, b in spans:
        assert np.array_equal(got[a:b], np.argsort(k[a:b], kind="stable")), (a, b)


@pytest.mark.parametrize("lens", [LONG, SHORT])
def test_outputs_of_freed_batches(ctx, lens):
    k, spans = column(lens, 3)
    dk = ctx.upload(k)
    keys = ctx.batch([dk.slice(a, b) for a, b in spans])
    orders = []
    for _ in range(12):  # every order stays alive, its batch does not
        order = ctx.upload(np.full(len(k), -1))
        ctx.batch_argsort(keys, ctx.batch([order.slice(a, b) for a, b in spans]))
        orders.append(order)
    for order in orders:
        check(order, k, spans)


@pytest.mark.parametrize("lens", [LONG, SHORT])
def test_captured_outputs_among_others(ctx, lens):
    k, spans = column(lens, 5)
    dk = ctx.upload(k)
    keys = ctx.batch([dk.slice(a, b) for a, b in spans])
    orders = [ctx.upload(np.full(len(k), -1)) for _ in range(9)]
    outs = [ctx.batch([o.slice(a, b) for a, b in spans]) for o in orders]
    ctx.batch_argsort(keys, outs[0], 0b11)
    ctx.synchronize()
    ctx.graph_begin()
    ctx.batch_argsort(keys, outs[0], 0b10000011)
    g = ctx.graph_end()
    for o in outs[1:]:
        ctx.batch_argsort(keys, o)
    ctx.elementwise_tile("sub_i64", [orders[0], orders[0]], orders[0])
    g.launch()
    for o in orders:
        check(o, k, spans)


def test_scratch_that_cannot_be_allocated():
    import verkehrt_gb300 as vk

    c = vk.Context(0)
    try:
        k, spans = column(LONG, 9)
        dk, first, second = c.upload(k), c.new_array("i64", len(k)), c.new_array("i64", len(k))
        keys = c.batch([dk.slice(a, b) for a, b in spans])
        outs = [c.batch([o.slice(a, b) for a, b in spans]) for o in (first, second)]
        for at in range(7):
            c.tune_set("fail_alloc_after", 0, at)
            with pytest.raises(vk.KernelError) as e:
                c.batch_argsort(keys, outs[0])
            assert e.value.status == "ALLOC"
        for o, out in ((first, outs[0]), (second, outs[1]), (first, outs[0])):
            c.batch_argsort(keys, out)
            check(o, k, spans)
    finally:
        c.close()
