"""Steps of single tokens: the kernels that stream weights and cached keys, at the edges of what they take."""

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_vedadra import context_for, step_of        # noqa: E402


@pytest.mark.parametrize("T,E,top,N,K", [(31, 16, 2, 2048, 2048),       # groups of several sizes
                                         (40, 2, 2, 1016, 1000),        # far more than eight pairs an expert, features and K with remainders
                                         (70, 5, 2, 264, 2056),         # more pairs than a launch takes
                                         (9, 4, 3, 250, 8200),          # long rows: groups of two pairs
                                         (6, 1, 1, 2100, 4096)])        # one group, rows held for one group at a time
@pytest.mark.parametrize("form", ["gate", "act", "plain"])
def test_the_grouped_stream_of_a_few_pairs(T, E, top, N, K, form):
    """Against the same operands in 64 bits.  A float32 sum of K products in any order is off by at most K 2^-24 of the
    sum of their sizes (far less in practice: 2^-17 is stated); a bfloat16 result by 2^-8 of itself more."""
    from ayaka_py_b200 import ops
    assert T * top * N * K >= 20 << 20                   # the grouped kernel's side of the line
    gen = torch.Generator(device="cuda").manual_seed(T + N)
    pairs, first = T * top, form != "plain"
    a = torch.randn(T if first else pairs, K, generator=gen, device="cuda").to(torch.bfloat16)
    w = (torch.randn(E, 2 * N if form == "gate" else N, K, generator=gen, device="cuda") / K ** 0.5).to(torch.bfloat16)
    route = ops.moe_route(torch.randn(T, E, generator=gen, device="cuda") * 2, E, top, plan=False)
    glu = (1.5, 1.702, 1.0) if form == "gate" else None
    got = ops.moe_gemv(a, w, route, glu=glu, activation="relu2" if form == "act" else None, weigh_input=form == "gate").double()
    x = a.double()
    for p in range(pairs):
        t, k = divmod(p, top)
        row, m = x[t if first else p], w[int(route.ids[t, k])].double()
        z, size = m @ row, m.abs() @ row.abs()
        if form == "gate":
            z, size = z * float(route.weights[t, k]), size * float(route.weights[t, k])
            g, u = z[:N].clamp(max=1.5), z[N:].clamp(-1.5, 1.5)
            want, room = g * torch.sigmoid(1.702 * g) * (u + 1.0), (size[:N] * 2.5 * 1.5 + size[N:] * 1.5)
        elif form == "act":
            want, room = z.clamp(min=0.0) ** 2, 2 * z.abs() * size
        else:
            want, room = z, size
        assert ((got[p] - want).abs() <= room * 2.0 ** -17 + (want.abs() * 2.0 ** -8 if first else 0.0) + 1e-6).all(), p
    assert ops.tc_error() == 0


@pytest.mark.parametrize("H,G,D,page,window,keep,chunk,cut", [
    (16, 4, 128, 16, None, 0, None, True), (8, 1, 128, 32, None, 0, None, True), (6, 2, 128, 16, 70, 9, None, True),
    (16, 2, 64, 64, 300, 0, None, True), (8, 4, 128, 16, None, 0, 100, True), (4, 4, 64, 16, 1, 0, None, True), (16, 4, 128, 16, None, 0, None, False)])
def test_single_rows_of_heads_that_share_their_keys(H, G, D, page, window, keep, chunk, cut):
    """The tensor-core kernel against the FP32 pipes on the same bfloat16 pages: contexts that end at the edges of the warps'
    16 keys and of partitions, a window far into a part, windows, kept first keys, chunks, sinks, gates."""
    from ayaka_py_b200 import ops
    from ayaka_py_b200.cache import CacheGroupSpec
    from ayaka_py_b200.parts.base import KVNeed
    torch.manual_seed(H + D)
    need = KVNeed(kv_heads=G, head_dim=D, window=window if not chunk else None, value_heads=G, value_dim=D, keep_first=keep if window else 0)
    before = [0, 1, 15, 16, 17, 63, 64, 127, 128, 255, 256, 511, 1000] if cut else [0, 15, 16, 63]
    cache, runner = context_for([CacheGroupSpec("g", need, 1)], "bfloat16", max_requests=len(before), page_size=page,
                                pages=sum(-(-(n + 1) // page) for n in before) + 2, positions=1024 if cut else 64)
    kpages, vpages = cache.kv_layer(0, 0)
    kpages.copy_(torch.randn(kpages.shape, device="cuda") * 0.7)
    vpages.copy_(torch.randn(vpages.shape, device="cuda"))
    for i, n in enumerate(before):
        slot = cache.open(i)
        if n:
            cache.commit(cache.reserve([(slot, 0, n)]))
    ctx, res = step_of(cache, runner, {i: 1 for i in range(len(before))})
    q = (torch.randn(ctx.num_rows, H * D, device="cuda") * 0.3).to(torch.bfloat16)
    for sinks, slopes in ((torch.randn(H, device="cuda"), None), (None, torch.rand(H, device="cuda") * 0.05)):
        kw = dict(heads=H, key_heads=G, key_dim=D, scale=0.6, window=window, keep_first=keep, chunk=chunk, sinks=sinks, slopes=slopes,
                  gate=torch.randn(ctx.num_rows, H * D, device="cuda"))
        got = ops.grouped_attention(q, kpages, vpages, ctx.tables[0], ctx, tensor_cores=True, **kw).float()
        want = ops.grouped_attention(q, kpages, vpages, ctx.tables[0], ctx, tensor_cores=False, **kw).float()
        assert torch.isfinite(got).all()
        # the weights enter the second product as bfloat16 (2^-9 of each), the result is rounded to bfloat16 twice
        assert float((got - want).abs().max()) < 1.5e-2 * float(want.abs().max())
    cache.rollback(res)


def test_more_choices_a_row_than_a_grouped_launch_holds():
    """Routes that a caller made: 130 experts a row."""
    from ayaka_py_b200 import ops
    T, top, N, K = 2, 130, 256, 512
    assert T * top * N * K >= 20 << 20
    gen = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randn(T, K, generator=gen, device="cuda").to(torch.bfloat16)
    w = (torch.randn(top, N, K, generator=gen, device="cuda") / K ** 0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(top, generator=gen, device="cuda") for _ in range(T)]).to(torch.int32)
    route = ops.MoeRoute(ids, torch.ones(T, top, device="cuda"), None, None, 0, top)
    got = ops.moe_gemv(a, w, route, glu=None, activation="relu2").double().view(T, top, N)
    want = torch.einsum("tk,tenk->ten", a.double(), w.double()[ids.long()]).clamp(min=0.0) ** 2
    assert bool(((got - want).abs() <= want * 2.0 ** -8 + 1e-5).all())
