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


# at most four rows per expert on average: none, one, a whole pass of eight, one more, several passes; k with a last step that
# lacks pieces, k shorter than a step of every warp, n with a remainder of 32 rows
@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[0, 1, 8, 9, 0, 0], [3] * 40, [40] + [0] * 11, [1]])
@pytest.mark.parametrize("n,k", [(16, 32), (1536, 2048), (40, 72), (8, 8), (24, 1000), (2048, 1536)])
def test_grouped_products_of_few_rows(counts, n, k):
    g = torch.Generator(device=DEV).manual_seed(n + k + len(counts))
    rows, experts, tokens = sum(counts), len(counts), 11
    off = torch.tensor([sum(counts[:i]) for i in range(experts + 1)], dtype=torch.int32, device=DEV)
    w = (torch.randn(experts, n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    x = torch.randn(tokens, k, generator=g, device=DEV).bfloat16()
    src = torch.randint(0, tokens, (rows,), generator=g, device=DEV).int()
    for gathered in (True, False):
        a = x if gathered else x[src.long()].contiguous()
        out = torch.full((rows + 2, n), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.moe_gemm(a, w, off, out[:rows], src=src if gathered else None, act="gelu" if gathered else "none")
        for e in range(experts):
            at = slice(int(off[e]), int(off[e + 1]))
            want = x[src[at].long()].double() @ w[e].double().t()
            if gathered:
                want = torch.nn.functional.gelu(want)
            # one rounding to bf16, and sums of k terms of size |x| |w| ~ 1 in fp32
            assert bool(((out[at].double() - want).abs() <= want.abs() * 2.0 ** -8 + k * 2.0 ** -22).all()), (e, gathered)
        assert bool((out[rows:] == 7.0).all())
