"""The tcgen05 attention of heads of 128 numbers (prompt portions) against the FP32 pipes, at the edges of its tiles of 128 rows and 64 keys."""

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_vedadra import context_for, step_of        # noqa: E402


@pytest.mark.parametrize("H,G,page,window,chunk", [
    (4, 2, 16, None, None),                                     # two heads of a key head share its tiles
    (3, 3, 8, None, None), (3, 1, 32, 70, None),                # 256 rows of one head to a block
    (8, 2, 128, None, 100), (4, 1, 256, 300, None), (5, 5, 16, None, 64), (2, 1, 16, 1, None), (2, 2, 64, None, 1)])
@pytest.mark.parametrize("before,brings", [
    ([0], [2]), ([0], [64]), ([0], [65]), ([0], [129]), ([0, 0], [256, 257]), ([63, 1000], [66, 300]), ([650, 17, 200], [1, 130, 2]), ([512], [511])])
def test_portions_on_tcgen05(H, G, page, window, chunk, before, brings):
    """Prompts and portions behind cached keys, single rows among them, windows, chunks, sinks, gates; the places behind a
    context's end hold infinities, which no row may see."""
    from ayaka_py_b200 import ops
    from ayaka_py_b200.cache import CacheGroupSpec
    from ayaka_py_b200.parts.base import KVNeed
    torch.manual_seed(H + page)
    D = 128
    need = KVNeed(kv_heads=G, head_dim=D, window=window, value_heads=G, value_dim=D)
    pages = sum(-(-(a + b) // page) for a, b in zip(before, brings)) + 2
    cache, runner = context_for([CacheGroupSpec("g", need, 1)], "bfloat16", max_requests=4, page_size=page, pages=pages, positions=2048)
    kpages, vpages = cache.kv_layer(0, 0)
    kpages.copy_(torch.randn(kpages.shape, device="cuda") * 0.7)
    vpages.copy_(torch.randn(vpages.shape, device="cuda"))
    for i, n in enumerate(before):
        slot = cache.open(i)
        if n:
            cache.commit(cache.reserve([(slot, 0, n)]))
    ctx, res = step_of(cache, runner, dict(enumerate(brings)))
    order = [int(r) for r in ctx.row_req.unique_consecutive()]
    ends = (ctx.req_pos0[:len(brings)] + (ctx.req_q_start[1:len(brings) + 1] - ctx.req_q_start[:len(brings)])).tolist()
    for r in order:
        last = ends[r] - 1
        cell = int(ctx.tables[0][r, last // page])
        kpages[cell, last % page + 1:] = float("inf")
        vpages[cell, last % page + 1:] = float("nan")
    T = ctx.num_rows
    q = (torch.randn(T, H * D, device="cuda") * 0.3).to(torch.bfloat16)
    gate = torch.randn(T, H * D + 8, device="cuda")
    for sinks, with_gate in ((None, None), (torch.randn(H, device="cuda"), gate)):
        kw = dict(heads=H, key_heads=G, key_dim=D, scale=0.6, window=window, chunk=chunk, sinks=sinks, gate=with_gate)
        got = ops.grouped_attention(q, kpages, vpages, ctx.tables[0], ctx, wide=True, **kw).float()
        want = ops.grouped_attention(q, kpages, vpages, ctx.tables[0], ctx, tensor_cores=False, **kw).float()
        assert ops.tc_error() == 0
        assert torch.isfinite(want).all() and torch.isfinite(got).all()
        # the weights enter the second product as bfloat16 (2^-9 of each), the result is rounded to bfloat16 on both sides
        assert float((got - want).abs().max()) < 1.5e-2 * float(want.abs().max())
    cache.rollback(res)
