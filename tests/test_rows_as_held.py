"""Log betas and positions of a prompt as the selection and the gather read them (``ops.rows_as_held``)."""
import pytest
import torch

from trimkv_b200 import ops


def _check(beta, pos, nseg, n, shared):
    b, p = ops.rows_as_held(beta, pos, nseg, n)
    assert b.shape == (nseg, n) and b.is_contiguous() and p.is_contiguous() and (p.dim() == 1) == shared
    assert torch.equal(b, beta.reshape(nseg, n)) and torch.equal(p.expand(nseg, n), pos.reshape(nseg, n))


@pytest.mark.parametrize("pos_type", [torch.int32, torch.int64])
def test_every_form_that_a_reshape_takes(pos_type):
    b, h, n = 2, 3, 5
    beta, line = torch.randn(b, h, n).bfloat16(), torch.arange(n, dtype=pos_type) + 4
    each = torch.arange(b * h * n, dtype=pos_type)
    _check(beta, line[None, None].expand(b, h, n), b * h, n, True)
    _check(beta, each.view(b, h, n), b * h, n, False)
    _check(beta, each.view(b, h, n)[:, :1].expand(b, h, n), b * h, n, False)         # shared by the heads of a request only
    _check(beta, each.view(b, n, h).transpose(1, 2), b * h, n, False)
    _check(beta, each.view(b * h, n), b * h, n, False)
    _check(beta, each, b * h, n, False)
    _check(beta, torch.arange(2 * n, dtype=pos_type)[::2][None, None].expand(b, h, n), b * h, n, True)
    _check(beta[:1, :1], line[None, None], 1, n, True)
    _check(beta[:, :, :0], line[None, None, :0].expand(b, h, 0), b * h, 0, True)
    _check(beta[:0], line[None, None].expand(0, h, n), 0, n, False)                  # an empty batch


@pytest.mark.parametrize("shape", [(1, 1, 5), (2, 1, 5), (1, 3, 5), (5,), (2, 3, 4), (2, 3, 1)])
def test_positions_that_are_not_one_per_segment_and_token_are_refused(shape):
    with pytest.raises(RuntimeError, match="shape"):
        ops.rows_as_held(torch.randn(2, 3, 5), torch.zeros(shape, dtype=torch.int64), 6, 5)


def test_types_that_the_kernels_do_not_read():
    beta, pos = torch.randn(1, 1, 4), torch.arange(4)[None, None]
    assert ops.rows_as_held(beta.double(), pos, 1, 4) is None and ops.rows_as_held(beta, pos.float(), 1, 4) is None
    assert ops.rows_as_held(beta, pos.short(), 1, 4) is None
