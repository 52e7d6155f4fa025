"""Experts with few rows: router logits and grouped products of a decoding step."""
import pytest
import torch

from trimkv_b200 import ops

DEV = "cuda"


# both sides of the size up to which the warp-per-logit kernel is taken; widths with a remainder of a warp's round
@pytest.mark.gpu
@pytest.mark.parametrize("tokens,experts,width", [(1, 1, 8), (7, 36, 2048), (8, 36, 264), (9, 5, 1032), (33, 64, 2048), (227, 36, 512), (228, 36, 512), (0, 4, 64)])
def test_router_logits(tokens, experts, width):
    g = torch.Generator(device=DEV).manual_seed(tokens + width)
    x = torch.randn(tokens, width + 16, generator=g, device=DEV).bfloat16()[:, 8:8 + width]      # rows further apart than their width
    w = torch.randn(experts, width, generator=g, device=DEV).bfloat16()
    z = ops.moe_logits(x, w)
    assert z.dtype == torch.float32 and z.shape == (tokens, experts)
    want = x.double() @ w.double().t()
    # products of 8-bit significands are exact in fp32: only the sum of `width` of them rounds
    bound = (x.double().abs() @ w.double().abs().t()) * (width * 2.0 ** -24)
    assert bool(((z.double() - want).abs() <= bound + 1e-30).all())
