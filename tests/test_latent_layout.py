"""How a latent attention lays its weights out, on the CPU."""

import pytest

torch = pytest.importorskip("torch")

from ayaka_py_b200.parts.latent_attention import LatentAttention          # noqa: E402

H, RANK, WIDTH = 3, 64, 96


def a_layer():
    part = LatentAttention(WIDTH, H, 128, 64, 128, RANK, 0.07, 1e-6, {"base": 50000.0, "dims": 64}, dtype=torch.bfloat16, device="cpu")
    gen = torch.Generator().manual_seed(3)
    w = {name: (torch.randn(d.shape, generator=gen) / d.shape[-1] ** 0.5).to(torch.bfloat16) if len(d.shape) == 2 else torch.ones(d.shape)
         for name, d in part.tensors().items()}
    return part, w


@pytest.mark.parametrize("factor", [1e9, float("inf"), float("nan")])
def test_weights_that_float16_cannot_hold_leave_none_of_the_old_behind(factor):
    part, w = a_layer()
    part.bind({k: v.clone() for k, v in w.items()})
    assert part.up_weight is not None
    w["uv_weight"][5] *= factor
    part.bind({k: v.clone() for k, v in w.items()})
    assert part.up_weight is None
    assert torch.equal(part.uv_weight.nan_to_num(1.0), w["uv_weight"].nan_to_num(1.0))


def test_every_heads_keys_and_values_come_to_the_top_of_float16():
    """The factors are powers of two; the largest number that a head's matrix can make of a normed latent lies in [2^14, 2^15) with it."""
    part, w = a_layer()
    for name, head, factor in (("uk_weight", 1, 2.0 ** -24), ("uv_weight", 0, 2.0 ** -20), ("uv_weight", 2, 0.0)):
        w[name].view(H, 128, RANK)[head] *= factor
    w["down_norm"] = w["down_norm"] * -0.3
    part.bind({k: v.clone() for k, v in w.items()})
    up = torch.cat([w["uk_weight"], w["uv_weight"]]).double().view(2 * H, 128, RANK)
    most = up.norm(dim=2).amax(dim=1) * 0.3 * RANK ** 0.5
    scaled = most * part.up_scale.double()
    assert part.up_scale.dtype == torch.float32 and bool((torch.frexp(part.up_scale).mantissa == 0.5).all())
    assert float(part.up_scale[H + 2]) == 1.0 and float(most[H + 2]) == 0.0
    scaled[H + 2] = 2.0 ** 14
    assert bool((scaled >= 2.0 ** 14 * (1 - 1e-6)).all()) and bool((scaled < 2.0 ** 15 * (1 + 1e-6)).all())
    assert torch.equal(part.up_weight.double(), (up * part.up_scale.double()[:, None, None]).view(2 * H * 128, RANK))
    assert torch.equal(part.uk_weight, w["uk_weight"]) and torch.equal(part.uv_weight, w["uv_weight"])           # ... of the other form


@pytest.mark.parametrize("factor,kept", [(2.0 ** -24, True), (2.0 ** -45, False), (1e-30, False)])
def test_a_head_too_small_for_its_factor_leaves_the_layer_unexpanded(factor, kept):
    part, w = a_layer()
    w["uk_weight"].view(H, 128, RANK)[1] *= factor
    part.bind(w)
    assert (part.up_weight is not None) is kept
