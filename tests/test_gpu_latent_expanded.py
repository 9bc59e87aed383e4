"""The latent attention with keys and values expanded against the same in 64 bits, beside the form that never expands them."""

import math
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_vedadra import context_for, step_of        # noqa: E402

RANK, ROT, DIM = 256, 64, 128


def reference(x, w, H, rot, window, gate, start_rows):
    """float64 rows of a whole sequence x [n, width]; the rows from start_rows on are returned."""
    n = x.shape[0]
    x = x.double()
    q = (x @ w["q_weight"].double().T).view(n, H, DIM + ROT)
    down = x @ w["down_weight"].double().T
    c, kr = down[:, :RANK], down[:, None, RANK:]
    c = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-6) * w["down_norm"].double()
    freq = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=torch.float64, device=x.device) / rot["dims"])
    angle = torch.arange(n, dtype=torch.float64, device=x.device)[:, None] * freq

    def turn(v):
        co, si = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
        out, d = v.clone(), rot["dims"]
        a, b = (slice(0, d // 2), slice(d // 2, d)) if rot["layout"] == "halves" else (slice(0, d, 2), slice(1, d, 2))
        out[..., a], out[..., b] = v[..., a] * co - v[..., b] * si, v[..., b] * co + v[..., a] * si
        return out

    qr, kr = turn(q[..., DIM:]), turn(kr)[:, 0]
    k = torch.einsum("nr,hdr->nhd", c, w["uk_weight"].double().view(H, DIM, RANK))
    v = torch.einsum("nr,hdr->nhd", c, w["uv_weight"].double().view(H, DIM, RANK))
    i, j = torch.arange(n, device=x.device)[:, None], torch.arange(n, device=x.device)[None]
    seen = (j <= i) & (i - j < (window or n + 1))
    out = torch.empty(n, H, DIM, dtype=torch.float64, device=x.device)
    for h in range(H):
        s = ((q[:, h, :DIM] @ k[:, h].T + qr[:, h] @ kr.T) * (DIM + ROT) ** -0.5).masked_fill(~seen, -math.inf)
        out[:, h] = torch.softmax(s, dim=1) @ v[:, h]
    if gate:
        g = torch.sigmoid(x @ w["gate_weight"].double().T)
        out = out * (g[:, :, None] if gate == "head" else g.view(n, H, DIM))
    return (out.reshape(n, H * DIM) @ w["out_weight"].double().T)[start_rows:]


@pytest.mark.parametrize("H,page,window,gate,layout,dims,gain", [
    (2, 16, None, None, "halves", 64, 1.0), (5, 8, 70, "head", "interleaved", 64, 1.0), (1, 64, None, "element", "halves", 32, 1.0),
    (3, 128, 200, None, "interleaved", 16, 1.0),
    (2, 16, None, None, "halves", 64, 3e4)])                # queries far beyond float16's range
@pytest.mark.parametrize("before,brings", [([0], [2]), ([0], [65]), ([3, 300], [129, 257]), ([63, 64, 200], [1, 66, 2]), ([510], [5])])
def test_expanded_keys_and_values(monkeypatch, H, page, window, gate, layout, dims, gain, before, brings):
    from ayaka_py_b200 import ops
    from ayaka_py_b200.cache import CacheGroupSpec
    from ayaka_py_b200.parts.latent_attention import LatentAttention
    torch.manual_seed(H + page)
    width = 256
    rot = {"base": 50000.0, "dims": dims, "layout": layout}
    part = LatentAttention(width, H, DIM, ROT, DIM, RANK, (DIM + ROT) ** -0.5, 1e-6, rot, gate=gate, window=window, dtype=torch.bfloat16)
    w = {name: (torch.randn(d.shape, device="cuda") / d.shape[-1] ** 0.5).to(torch.bfloat16) if len(d.shape) == 2 else 1 + 0.1 * torch.randn(d.shape, device="cuda")
         for name, d in part.tensors().items()}
    w["q_weight"] *= gain
    part.bind(w)
    assert part.up_weight is not None
    cache, runner = context_for([CacheGroupSpec("g", part.cache_need(), 1)], "bfloat16", max_requests=4, page_size=page,
                                pages=sum(-(-(a + b) // page) for a, b in zip(before, brings)) + 2)
    binding = SimpleNamespace(group=0, layer=0, writes=True)
    rows = {i: torch.randn(a + b, width, device="cuda").to(torch.bfloat16) for i, (a, b) in enumerate(zip(before, brings))}
    monkeypatch.setattr(ops, "latent_expanded_pays", lambda *a: False)
    for i, n in enumerate(before):
        cache.open(i)
        if n:
            ctx, res = step_of(cache, runner, {i: n})
            part.forward(rows[i][:n], None, ctx, binding)
            cache.commit(res)
    ctx, res = step_of(cache, runner, dict(enumerate(brings)))
    plan = sorted(range(len(brings)), key=lambda i: brings[i] != 1)       # a step's single rows come first
    x = torch.cat([rows[i][before[i]:] for i in plan])
    want = torch.cat([reference(rows[i], w, H, rot, window, gate, before[i]) for i in plan])
    errors = []
    for expanded in (False, True):
        monkeypatch.setattr(ops, "latent_expanded_pays", lambda *a, e=expanded: e)
        got = part.forward(x, None, ctx, binding).double()
        assert torch.isfinite(got).all() and ops.tc_error() == 0
        errors.append(float((got - want).norm() / want.norm()))
    # bfloat16 products around the attention: 3e-3 on both sides; a far larger spread of the scores makes every rounding count for more
    assert errors[1] < (8e-3 if gain == 1.0 else 0.2), errors
    assert errors[1] < 1.2 * errors[0] + 1e-3, errors
    cache.rollback(res)


def a_layer(H, before, brings, window=None, page=16, scales=None):
    """(part, weights, context, packed rows, place of every request's rows) of a step that brings ``brings`` tokens behind ``before``; ``scales``:
    factors on the weights by name."""
    from ayaka_py_b200.cache import CacheGroupSpec
    from ayaka_py_b200.parts.latent_attention import LatentAttention
    torch.manual_seed(H + sum(brings))
    width = 256
    part = LatentAttention(width, H, DIM, ROT, DIM, RANK, (DIM + ROT) ** -0.5, 1e-6, {"base": 50000.0, "dims": ROT, "layout": "halves"}, gate="head",
                           window=window, dtype=torch.bfloat16)
    w = {name: (torch.randn(d.shape, device="cuda") / d.shape[-1] ** 0.5).to(torch.bfloat16) if len(d.shape) == 2 else 1 + 0.1 * torch.randn(d.shape, device="cuda")
         for name, d in part.tensors().items()}
    for name, factor in (scales or {}).items():
        w[name] = w[name] * factor
    part.bind(w)
    cache, runner = context_for([CacheGroupSpec("g", part.cache_need(), 1)], "bfloat16", max_requests=4, page_size=page,
                                pages=sum(-(-(a + b) // page) for a, b in zip(before, brings)) + 2)
    for pages in cache.kv_layer(0, 0):
        pages.copy_(torch.randn(pages.shape, device="cuda"))
    for i, n in enumerate(before):
        slot = cache.open(i)
        if n:
            cache.commit(cache.reserve([(slot, 0, n)]))
    ctx, _ = step_of(cache, runner, dict(enumerate(brings)))
    order = [int(i) for i in ctx.host["order"]]
    at = {i: slice(int(ctx.host["q_start"][k]), int(ctx.host["q_start"][k + 1])) for k, i in enumerate(order)}
    return part, w, ctx, torch.randn(ctx.num_rows, width, device="cuda").to(torch.bfloat16), at


@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("before,brings,bad", [([0, 0], [65, 70], 1), ([0, 0], [64, 64], 1), ([63, 10], [130, 257], 1), ([3, 300], [2, 5], 1),
                                               ([0, 0, 0], [700, 257, 33], 1), ([500, 40], [300, 2], 0)])
def test_a_request_that_is_no_number_keeps_to_itself(monkeypatch, before, brings, bad, window):
    """Keys and values lie request after request, and a tile of 64 of them holds the next request's first ones."""
    from ayaka_py_b200 import ops
    monkeypatch.setattr(ops, "latent_expanded_pays", lambda *a: True)
    part, _, ctx, x, at = a_layer(2, before, brings, window)
    binding = SimpleNamespace(group=0, layer=0, writes=True)
    want = part.forward(x, None, ctx, binding).clone()
    x[at[bad]] = math.inf
    got = part.forward(x, None, ctx, binding)
    assert ops.tc_error() == 0 and not torch.isfinite(got[at[bad]]).any()
    for i in range(len(brings)):
        if i != bad:
            assert torch.isfinite(want[at[i]]).all() and torch.equal(got[at[i]], want[at[i]]), i


def heads_of(monkeypatch, part, x, ctx):
    """The heads' outputs [T, H, 128] of the expanded form."""
    from ayaka_py_b200 import ops
    made, expanded = [], ops.latent_expanded
    monkeypatch.setattr(ops, "latent_expanded_pays", lambda *a: True)
    with monkeypatch.context() as m:
        m.setattr(ops, "latent_expanded", lambda *a: made.append(expanded(*a)) or made[-1])
        part.forward(x, None, ctx, SimpleNamespace(group=0, layer=0, writes=True))
    assert ops.tc_error() == 0
    return made[0].view(x.shape[0], part.heads, DIM).double()


@pytest.mark.parametrize("before,brings", [([0], [257]), ([70, 300], [129, 3])])
@pytest.mark.parametrize("power", [-24, -28, 9])
def test_a_heads_scale_is_not_its_precision(monkeypatch, before, brings, power):
    """U_v of one head times a power of two is its output times that, bit for bit; U_k times it and the queries divided by it change nothing."""
    H, head = 3, 1
    part, w, ctx, x, _ = a_layer(H, before, brings)
    want = heads_of(monkeypatch, part, x, ctx)
    values = {k: v.clone() for k, v in w.items()}
    values["uv_weight"].view(H, DIM, RANK)[head] *= 2.0 ** power
    part.bind(values)
    got = heads_of(monkeypatch, part, x, ctx)
    got[:, head] *= 2.0 ** -power
    assert part.up_weight is not None and torch.equal(got, want)
    keys = {k: v.clone() for k, v in w.items()}
    keys["uk_weight"].view(H, DIM, RANK)[head] *= 2.0 ** power
    keys["q_weight"].view(H, DIM + ROT, -1)[head, :DIM] *= 2.0 ** -power
    part.bind(keys)
    assert part.up_weight is not None and torch.equal(heads_of(monkeypatch, part, x, ctx), want)


def test_small_values_keep_their_bits(monkeypatch):
    """Values of 1e-7 lose 17 % in float16 without a factor; bounds as for ordinary ones."""
    part, w, ctx, x, _ = a_layer(2, [0], [300], scales={"uv_weight": 1e-7})
    from ayaka_py_b200 import ops
    monkeypatch.setattr(ops, "latent_expanded_pays", lambda *a: True)
    got = part.forward(x, None, ctx, SimpleNamespace(group=0, layer=0, writes=True)).double()
    want = reference(x, w, 2, {"base": 50000.0, "dims": ROT, "layout": "halves"}, None, "head", 0)
    assert part.up_weight is not None and float((got - want).norm() / want.norm()) < 8e-3


def test_small_weights_keep_their_bits():
    """One key takes all but 2e-9 of the weight and has a value of zero: what the others leave is the whole output.  Their weights
    are rounded to float16 (2^-11 of each), their values too, the output to bfloat16: 2^-8 of the whole."""
    from ayaka_py_b200 import ops
    from ayaka_py_b200.cache import CacheGroupSpec
    from ayaka_py_b200.parts.base import KVNeed
    torch.manual_seed(1)
    T = 200
    need = KVNeed(kv_heads=1, head_dim=ROT, value_heads=1, value_dim=RANK)
    cache, runner = context_for([CacheGroupSpec("g", need, 1)], "bfloat16", page_size=16, pages=20)
    ctx, _ = step_of(cache, runner, {0: T})
    rope, latent = cache.kv_layer(0, 0)
    proj = torch.zeros(T, DIM + ROT + RANK + ROT, device="cuda")
    proj[:, 0] = 1.25                                    # 20 with the first key
    down = proj[:, DIM + ROT:]
    down[0, 0] = 1.0                                     # the first latent: 16 in its first place
    down[1:, RANK // 2:RANK] = torch.randn(T - 1, RANK // 2, device="cuda")
    up = torch.zeros(2 * DIM, RANK, device="cuda")
    up[0, 0] = 1.0
    up[DIM:, RANK // 2:] = torch.randn(DIM, RANK // 2, device="cuda") / 16
    up = up.to(torch.bfloat16)
    factor = torch.tensor([512.0, 256.0], device="cuda")
    scaled = (up.view(2, DIM, RANK) * factor[:, None, None]).to(torch.bfloat16).view(2 * DIM, RANK)
    got = ops.latent_expanded(proj, latent, rope, scaled, factor, torch.ones(RANK, device="cuda"),
                              torch.zeros(1, device="cuda"), 1.0, 0, ctx, ctx.tables[0], 1, 1e-12, False, 1.0, None, None).double()
    c = down[:, :RANK].double()
    c = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-12)
    scores = (proj[:, :1].double() @ c[:, :1].T).masked_fill(torch.ones(T, T, device="cuda").triu(1).bool(), -math.inf)
    want = torch.softmax(scores, dim=1) @ (c @ up[DIM:].double().T)
    assert ops.tc_error() == 0 and float(want[1:].abs().max()) < 1e-6
    assert float((got[1:] - want[1:]).norm() / want[1:].norm()) < 2.0 ** -8
