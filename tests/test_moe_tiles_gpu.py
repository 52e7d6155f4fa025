"""Grouped products of few rows per expert (csrc/tkv_moe_tc.cu): tiles of 64 rows and stages of 128 columns of k, where k is of whole
pieces of 64; of other k, tiles of 128 rows and stages of 64 columns."""
import pytest
import torch

from trimkv_b200 import ops

pytestmark = pytest.mark.gpu


EDGES = [[1, 0, 63, 0, 64, 2, 0, 1], [0, 0, 150, 1, 0, 0, 65, 0]]


@pytest.mark.parametrize("k", [8, 64, 72, 128, 200, 456])
@pytest.mark.parametrize("counts", EDGES)
def test_rows_and_columns_at_the_edges_of_tiles(k, counts):
    """Experts without rows, with 64 and more than 64 (two tiles) of them; one stage of whole pieces or a part of one, and other k."""
    _check(k, counts, 4232)


@pytest.mark.parametrize("k,n", [(192, 16904), (320, 16904), (576, 16904), (1088, 16904), (2048, 8456)])
@pytest.mark.parametrize("counts", EDGES)
def test_stages_and_accumulators_are_used_again(k, counts, n):
    """More stages of 128 columns than the ring has, a half one behind whole ones, and more tiles per CTA than accumulators."""
    _check(k, counts, n)


def _check(k, counts, n):
    experts, rows = len(counts), sum(counts)
    tiles = sum(-(-c // 64) for c in counts) * -(-n // 128)
    assert rows <= 32 * experts and tiles > 148
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(40, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(experts, n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    off = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    src = torch.randint(0, 40, (rows,), generator=g, device="cuda", dtype=torch.int32)
    got = torch.full((rows + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.moe_gemm(x, w, off, got[:rows], src=src)
    plain = torch.full_like(got, 7.0)
    ops.moe_gemm(x[src.long()].contiguous(), w, off, plain[:rows])
    assert torch.equal(got, plain) and bool((got[rows] == 7.0).all())
    at = 0
    for e, c in enumerate(counts):
        want = x[src[at:at + c].long()].double() @ w[e].double().t()
        # one rounding to bf16 (2^-9), and fp32 sums of k products
        assert bool(((got[at:at + c].double() - want).abs() <= want.abs() * 2.0 ** -8 + k * 2.0 ** -22).all())
        at += c
