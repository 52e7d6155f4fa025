"""Query-resident attention with one and with two tiles of 128 query rows per CTA, at the edges of the tiles."""
import pytest
import torch

from trimkv_b200 import _lib, ops

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
# that end at, before and behind the edge of a key tile, and (40 of 130 tokens) ones of which the first rows see nothing.  Of 257 rows
# the last CTA's second tile has none, of 400 rows against 200 keys a CTA's first tile sees nothing and its second does.  Alone the
# segments are few: one tile per CTA; `copies` times over they are many: two.
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,ql,lens,copies", [
    (1, 1, 1, (1, 128, 129), 1), (2, 2, 128, (128, 256, 383, 200), 1), (3, 1, 43, (300, 43), 40), (2, 1, 128, (128, 129, 640), 27),
    (1, 1, 257, (257, 258, 512), 24), (1, 1, 130, (40, 130, 131), 27), (4, 2, 64, (64, 127, 500, 65), 1), (4, 2, 65, (65, 127, 500, 66), 20),
    (3, 3, 385, (385, 512, 700), 14), (1, 1, 400, (200, 400), 37), (1, 1, 300, (20, 170, 172), 24),
])
def test_tile_edges(dtype, hq, hkv, ql, lens, copies):
    g = torch.Generator(device=DEV).manual_seed(hq + 10 * ql)
    b, cap, d = len(lens) // hkv, max(max(lens), 150), 128
    q = torch.randn(b, ql, hq, d, generator=g, device=DEV).to(dtype)
    k = torch.randn(len(lens), cap, d, generator=g, device=DEV).to(dtype)
    v = torch.randn(len(lens), cap, d, generator=g, device=DEV).to(dtype)
    k[0, 0] *= 6.0                             # a maximum that grows late or early: sums are rescaled
    k[-1, lens[-1] - 1] *= 8.0
    for s, n in enumerate(lens):               # what lies behind a segment must not leak
        k[s, n:], v[s, n:] = float("nan"), float("inf")
    want = _reference(q, k, v, lens, hkv, d ** -0.5)
    # weights and result are rounded to the 16-bit type: an error of each weight of half a unit against values of up to 4.5
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    outs = []
    for times in sorted({1, copies}):
        assert _lib.lib().tkv_prefill_attn_rows_per_cta(len(lens) * times, ql * hq // hkv) == (128 if times == 1 else 256)
        out = torch.full((b * times, ql, hq, d), float("nan"), dtype=dtype, device=DEV)
        status = ops.new_status(DEV)
        ops.prefill_attn(q.repeat(times, 1, 1, 1), k.repeat(times, 1, 1), v.repeat(times, 1, 1),
                         torch.tensor(lens * times, dtype=torch.int32, device=DEV), cap, out, hkv, d ** -0.5, cap, status)
        assert ops.read_status(status) == 0
        outs.append(out)
        assert (out.view(times, b, ql, hq, d).double() - want).abs().max().item() <= 4.5 * unit + unit
    assert torch.equal(outs[-1].view(-1, *outs[0].shape), outs[0].expand(copies, *outs[0].shape))     # the same sums in the same order


@pytest.mark.gpu
@pytest.mark.parametrize("n,copies", [(129, 40), (256, 40), (257, 27), (400, 36), (511, 36)])
@pytest.mark.parametrize("window", [1, 127, 128, 129, 300, 5000])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (40, 24)])
def test_two_part_keys(n, copies, window, dim, vdim):
    """One request (one tile per CTA) and many of it (two): against 64 bits, and the same bit for bit."""
    from tests.test_dafovik_gpu import cache_of
    from trimkv_b200.state_cache import LatentState
    g = torch.Generator(device=DEV).manual_seed(n + window)
    heads, rot, rank, scale = 2, 64, 64, 0.11
    q = torch.randn(n, heads * (dim + rot), generator=g, device=DEV).bfloat16()
    kv = torch.randn(n, heads * (dim + vdim), generator=g, device=DEV).bfloat16()
    lin = torch.randn(n, rank + rot, generator=g, device=DEV).bfloat16()
    outs = []
    for times in (1, copies):
        assert _lib.lib().tkv_latent_prefill_rows_per_cta(times, heads, n * times, n) == (128 if times == 1 else 256)
        cache = cache_of(LatentState(rank + rot, window), dtype=torch.bfloat16)
        cache.open(times)
        b = cache.begin([n] * times)
        out = torch.full((n * times, heads * vdim), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.latent_prefill(q.repeat(times, 1), kv.repeat(times, 1), lin.repeat(times, 1), b, scale, out, heads, dim, rot, vdim, rank, window)
        cache.check_status()
        outs.append(out.view(times, n, -1))
    assert torch.equal(outs[1], outs[0].expand_as(outs[1]))
    gap = torch.arange(n, device=DEV)[:, None] - torch.arange(n, device=DEV)
    q3, k3 = q.view(n, heads, -1).double(), kv[:, :heads * dim].reshape(n, heads, dim).double()
    v3 = kv[:, heads * dim:].reshape(n, heads, vdim).double()
    s = (torch.einsum("ihd,jhd->hij", q3[..., :dim], k3) + torch.einsum("ihd,jd->hij", q3[..., dim:], lin[:, rank:].double())) * scale
    want = torch.einsum("hij,jhp->ihp", s.masked_fill((gap < 0) | (gap >= window), float("-inf")).softmax(-1), v3)
    # weights and result rounded to bf16, values of up to 4.5
    assert (outs[0][0].double() - want.reshape(n, -1)).abs().max().item() <= 5.5 * 2.0 ** -8
