"""Query-resident attention with two tiles of 128 query rows per CTA, at the edges of the tiles."""
import pytest
import torch

from trimkv_b200 import ops

DEV = "cuda"


def _reference(q, k, v, lens, hkv, scale):
    """64-bit attention; row i of a segment of n tokens sees the first n - Q + i + 1, a row that sees nothing is zero."""
    b, ql, hq, d = q.shape
    group = hq // hkv
    out = torch.zeros(q.shape, dtype=torch.float64, device=q.device)
    for s, n in enumerate(lens):
        i, h = divmod(s, hkv)
        heads = slice(h * group, (h + 1) * group)
        for t in range(ql):
            m = n - ql + t + 1
            if m > 0:
                w = (q[i, t, heads].double() @ k[s, :m].double().T * scale).softmax(-1)
                out[i, t, heads] = w @ v[s, :m].double()
    return out


# rows of a segment = q_tokens * hq / hkv: one tile, its edge, one row into the second, both, one row into the next CTA; segments
# that end at, before and behind the edge of a key tile, and (40 of 130 tokens) ones of which the first rows see nothing
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,ql,lens", [
    (1, 1, 1, (1, 128, 129)), (2, 2, 128, (128, 256, 383, 200)), (3, 1, 43, (300, 43)), (2, 1, 128, (128, 129, 640)),
    (1, 1, 257, (257, 258, 512)), (1, 1, 130, (40, 130, 131)), (4, 2, 64, (64, 127, 500, 65)), (3, 3, 385, (385, 512, 700)),
])
def test_tile_edges(dtype, hq, hkv, ql, lens):
    g = torch.Generator(device=DEV).manual_seed(hq + 10 * ql)
    b, cap, d = len(lens) // hkv, max(max(lens), 150), 128
    q = torch.randn(b, ql, hq, d, generator=g, device=DEV).to(dtype)
    k = torch.randn(len(lens), cap, d, generator=g, device=DEV).to(dtype)
    v = torch.randn(len(lens), cap, d, generator=g, device=DEV).to(dtype)
    k[0, 0] *= 6.0                             # a maximum that grows late or early: sums are rescaled
    k[-1, lens[-1] - 1] *= 8.0
    for s, n in enumerate(lens):               # what lies behind a segment must not leak
        k[s, n:], v[s, n:] = float("nan"), float("inf")
    out = torch.full(q.shape, float("nan"), dtype=dtype, device=DEV)
    status = ops.new_status(DEV)
    ops.prefill_attn(q, k, v, torch.tensor(lens, dtype=torch.int32, device=DEV), cap, out, hkv, d ** -0.5, cap, status)
    assert ops.read_status(status) == 0
    want = _reference(q, k, v, lens, hkv, d ** -0.5)
    # weights and result are rounded to the 16-bit type: an error of each weight of half a unit against values of up to 4.5
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert (out.double() - want).abs().max().item() <= 4.5 * unit + unit
