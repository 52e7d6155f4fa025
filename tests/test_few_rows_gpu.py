"""The product of a few rows (csrc/tkv_few_rows.cu) against fp64, and where ``ops.linear`` takes it."""
import pytest
import torch
import torch.nn.functional as F

from trimkv_b200 import ops
from trimkv_b200._lib import lib

pytestmark = pytest.mark.gpu


def _near(y, x, w, bias=None):
    """One rounding to bf16 (2^-8 of the value, which allows for the neighbour) and fp32 sums of k products."""
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    if bias is not None:
        want, size = want + bias.double(), size + bias.double().abs()
    return bool(((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * x.shape[1] * 2.0 ** -24).all())


@pytest.mark.parametrize("m", [1, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(8, 64), (128, 128), (136, 192), (1000, 320), (2048, 9216), (5120, 1088), (33000, 64)])
def test_tiles_rows_and_pieces(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(n + m)
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    bias = torch.randn(n, generator=g, device="cuda").bfloat16()
    status = ops.new_status(x.device)
    for b in (None, bias):
        y = torch.full((m * n + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
        assert lib().tkv_few_rows(x.data_ptr(), w.data_ptr(), ops._ptr(b), y.data_ptr(), m, n, k, status.data_ptr(), ops._stream(x)) == 0
        assert _near(y[:m * n].view(m, n), x, w, b) and bool((y[m * n:] == 7.0).all()) and ops.read_status(status) == 0


def test_what_is_not_finite_stays_in_its_row_and_column():
    x, w = torch.ones(3, 1024, device="cuda").bfloat16(), torch.ones(256, 1024, device="cuda").bfloat16()
    x[1, 700], w[130, 3] = float("inf"), float("nan")
    y, want = ops.linear(x, w), F.linear(x, w)
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf()) and float(y[0, 0]) == 1024.0


def test_other_forms_go_to_the_library():
    """Whatever the kernel does not take gives what the library gives, bit for bit; what the library refuses stays refused."""
    x, w = torch.randn(4, 1024, device="cuda"), torch.randn(256, 1024, device="cuda")
    xb, wb = x.bfloat16(), w.bfloat16()
    calls = [(x, w), (x.half(), w.half()), (xb[:, ::2], wb[:, ::2]), (xb.view(2, 2, 1024), wb), (xb[0], wb), (xb[:0], wb),
             (torch.randn(33, 1024, device="cuda").bfloat16(), wb), (xb, torch.randn(5128, 1024, device="cuda").bfloat16()),
             (xb, wb[:255]), (xb[:, :1000], wb[:, :1000]), (xb[:, :960].contiguous(), wb[:, :960].contiguous()), (xb.cpu(), wb.cpu())]
    with torch.no_grad():
        for a, b in calls:
            assert torch.equal(ops.linear(a, b), F.linear(a, b)), (a.shape, b.shape)
        for b in (torch.randn(256, device="cuda").bfloat16(), torch.randn(512, device="cuda").bfloat16()[::2], torch.randn(257, device="cuda").bfloat16()[1:]):
            assert (ops.linear(xb, wb, b).float() - F.linear(xb, wb, b).float()).abs().max() <= 2.0      # a step of values up to 256
        assert torch.equal(ops.linear(x, w, x[0, :256]), F.linear(x, w, x[0, :256]))
    p = wb.clone().requires_grad_()
    ops.linear(xb, p).sum().backward()
    assert p.grad is not None
    for a, b, c in ((xb, w, None), (xb, wb[:, :1016], None), (xb.cpu(), wb, None), (xb, wb, wb[0]), (xb, wb, x[0, :256])):
        with pytest.raises(RuntimeError):
            ops.linear(a, b, c)


def test_captured_with_the_kernel_before_and_after():
    """Recorded behind a kernel that writes its input and before one that reads its result; the weights change between replays."""
    u = torch.randn(8, 2048, device="cuda").bfloat16()
    x, w = u.clone(), torch.randn(2048, 2048, device="cuda").bfloat16() * 2048 ** -0.5

    def step():
        x.copy_(u)
        ops.gelu_tanh(x)
        y = ops.linear(x, w)
        ops.gelu_tanh(y)
        return y

    with torch.no_grad():
        want = step().clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = step()
        for sign in (1, -1):
            w.mul_(sign)
            graph.replay()
            assert torch.equal(y, want if sign == 1 else step())
