"""The experts' products of many rows: the activation in the first product's epilogue, and only the tiles that hold rows."""

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,top,d,inner", [(1, 4, 1, 64, 8), (64, 16, 2, 128, 72), (257, 3, 2, 136, 264), (700, 5, 4, 256, 1000), (129, 1, 1, 64, 136)])
@pytest.mark.parametrize("limit,weigh", [(float("inf"), True), (1.25, False)])
def test_experts_of_many_rows(T, E, top, d, inner, limit, weigh):
    """Against the same operands in 64 bits: the hidden rows are rounded to bfloat16 once (2^-9 of each, of random sign in the second sum)."""
    from ayaka_py_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(T + inner)
    h = torch.randn(T, d, generator=gen, device="cuda").to(torch.bfloat16)
    w1 = (torch.randn(E, 2 * inner, d, generator=gen, device="cuda") / d ** 0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, d, inner, generator=gen, device="cuda") / inner ** 0.5).to(torch.bfloat16)
    logits = torch.randn(T, E, generator=gen, device="cuda")
    logits[:, E - 1] += 3.0                              # one expert takes most rows, others few or none
    route = ops.moe_route(logits, E, top, plan=False)
    picked, rows = ops.moe_experts_tc(h, w1, w2, route, limit, 1.702, 0.5, weigh_input=weigh)
    assert ops.tc_error() == 0
    got = picked[rows.long()].double().view(T, top, d)
    want = torch.empty_like(got)
    for e in range(E):
        t, k = torch.nonzero(route.ids == e, as_tuple=True)
        x = h[t].double() @ w1[e].double().T
        if weigh:
            x = x * route.weights[t, k].double()[:, None]
        g, u = x[:, :inner].clamp(max=limit), x[:, inner:].clamp(-limit, limit)
        want[t, k] = (g * torch.sigmoid(1.702 * g) * (u + 0.5)) @ w2[e].double().T
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8
    assert float((got - want).abs().max()) < 2.0 ** -6 * float(want.abs().max())
