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
