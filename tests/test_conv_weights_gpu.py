"""The convolution's weights as vectors (csrc/tkv_linrec.cu): weights that start between two vectors give the same bits, by a channel or
(16-bit inputs of many tokens) eight channels per thread."""
import pytest
import torch

from trimkv_b200 import ops
from trimkv_b200.state_cache import HybridStateCache, RecurrentState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("channels,lens", [(8, [1, 33]), (1032, [31, 64, 5]), (1028, [40]), (2056, [3000, 1801])])
def test_aligned_and_shifted_weights_agree(channels, lens, dtype):
    g = torch.Generator(device="cuda").manual_seed(channels)
    x = torch.randn(sum(lens), channels, generator=g, device="cuda").to(dtype)
    w, bias = torch.randn(channels, 4, generator=g, device="cuda"), torch.randn(channels, generator=g, device="cuda")
    shifted = torch.empty(channels * 4 + 1, device="cuda")[1:].view(channels, 4).copy_(w)
    assert w.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 4
    got = []
    for weights in (w, shifted):
        cache = HybridStateCache([RecurrentState(1, 8, 8)], torch.device("cuda"), dtype)
        cache.open(len(lens))
        ring = torch.zeros(len(lens), 4, channels, device="cuda", dtype=dtype)
        out = torch.empty_like(x)
        ops.conv_silu(x, ring, weights, bias, out, cache.begin(list(lens)))
        got.append((out, ring))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    at = 0
    for n in lens:
        rows = torch.cat([torch.zeros(3, channels, device="cuda", dtype=torch.float64), x[at:at + n].double()])
        z = bias.double() + sum(w[:, k].double() * rows[k:k + n] for k in range(4))
        # four fp32 products, the hardware's exponential and division (2^-20), one rounding of the result
        near = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -18
        assert bool(((got[0][0][at:at + n].double() - z * torch.sigmoid(z)).abs() <= z.abs() * near + near * 2.0 ** -2).all())
        at += n
