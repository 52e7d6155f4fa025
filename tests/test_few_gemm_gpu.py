"""Projections of few rows."""
import pytest
import torch
import torch.nn.functional as F

from trimkv_b200 import _lib, ops

DEV = "cuda"


# edges of the tiles of 8 rows of x and of 16 and 32 of w (32 from 4737 on); k shorter than a step of every warp, with a last step
# that lacks pieces, longer than the ring
@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(16, 32), (1, 8), (40, 72), (2112, 2048), (17, 1000), (264, 6144), (4736, 136), (4737, 136), (8216, 2048)])
def test_products(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x = torch.randn(m, k + 16, generator=g, device=DEV).bfloat16()[:, 8:8 + k]                # rows further apart than their width
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    out = torch.full((m + 1, n + 3), 7.0, dtype=torch.bfloat16, device=DEV)
    _lib.check(_lib.lib().tkv_few_gemm(x.data_ptr(), x.stride(0), w.data_ptr(), out.data_ptr(), n + 3, m, n, k, ops.dtype_code(x.dtype),
                                       torch.cuda.current_stream().cuda_stream), "tkv_few_gemm")
    want = x.double() @ w.double().t()
    # one rounding to bf16, and the sum of k exact products in fp32
    bound = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * (k * 2.0 ** -24) + 1e-30
    assert bool(((out[:m, :n].double() - want).abs() <= bound).all())
    assert bool((out[m:] == 7.0).all()) and bool((out[:, n:] == 7.0).all())


@pytest.mark.gpu
def test_what_the_rule_leaves_to_the_library():
    x, w = torch.randn(4, 64, device=DEV).bfloat16(), torch.randn(24, 64, device=DEV).bfloat16()
    wide = torch.randn(ops.FEW_COLUMNS + 1, 64, device=DEV).bfloat16()
    before = ops.launch_count
    many = x.repeat(5, 1)
    for a, b in ((x.float(), w.float()), (x[:0], w), (many, w), (x, wide), (x[:, 1:41], w[:, :40].contiguous()), (x, w.t().contiguous().t()), (x[None], w)):
        assert torch.equal(ops.linear(a, b), F.linear(a, b))
    assert ops.linear(x, w.clone().requires_grad_()).requires_grad
    assert ops.launch_count == before
    with torch.no_grad():
        ops.linear(x, torch.nn.Parameter(w))
    assert ops.launch_count == before + 1
