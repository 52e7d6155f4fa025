"""Eviction by CTAs of 1024, 512 and 256 threads: on both sides of the numbers of segments where the width changes."""
import pytest
import torch

from trimkv_b200 import ops

DEV = "cuda"


# lengths with a remainder of a round of either width; 600 rows kept: several tiles of rows, the last one short
@pytest.mark.gpu
@pytest.mark.parametrize("nseg", [1, 148, 149, 296, 297])
@pytest.mark.parametrize("n,m", [(1541, 600), (1025, 1024), (300, 7)])
def test_widths_agree(nseg, n, m):
    g = torch.Generator(device=DEV).manual_seed(nseg + n)
    cap, d = n + 3, 64
    k, v = (torch.randn(nseg * cap, d, generator=g, device=DEV).bfloat16() for _ in range(2))
    beta = -torch.rand(nseg * cap, generator=g, device=DEV).mul(8).round().div(8)             # many equal scores ..
    beta.view(nseg, cap)[:, ::3] -= torch.rand(nseg, -(-cap // 3), generator=g, device=DEV)   # .. among others
    pos = torch.arange(cap, dtype=torch.int32, device=DEV).repeat(nseg)
    score = beta.view(nseg, cap)[:, :n] * (n + 1 - pos[:n]).float()
    keep = score.sort(dim=1, descending=True, stable=True).indices[:, :m].sort(dim=1).values
    kept, count = torch.empty(nseg, m, dtype=torch.int32, device=DEV), torch.empty(nseg, dtype=torch.int32, device=DEV)
    ops.evict_select(beta.view(nseg, cap), pos[:cap], None, n, nseg, n + 1, m, m, n, kept, count)
    assert torch.equal(kept.long(), keep) and bool((count == m).all())
    want = [t.view(nseg, cap, -1).gather(1, keep[:, :, None].expand(-1, -1, t.numel() // (nseg * cap))) for t in (k, v, beta, pos)]
    ln = torch.full((nseg,), n, dtype=torch.int32, device=DEV)
    status = ops.new_status(DEV)
    ops.evict(k, v, beta, pos, ln, None, nseg, nseg, cap, n + 1, m, m, n, status=status)
    assert ops.read_status(status) == 0 and bool((ln == m).all())
    for t, w in zip((k, v, beta, pos), want):
        assert torch.equal(t.view(nseg, cap, -1)[:, :m], w)


# log betas in every type, positions in 32 and 64 bits, shared by all segments and not; a prompt that is reduced and one that is not
@pytest.mark.gpu
@pytest.mark.parametrize("beta_type", [torch.float32, torch.bfloat16, torch.float16, torch.float64])
@pytest.mark.parametrize("pos_type,shared", [(torch.int64, True), (torch.int32, True), (torch.int64, False), (torch.int32, False)])
@pytest.mark.parametrize("n,transposed", [(333, False), (333, True), (120, False)])
def test_prompts_in_the_callers_types(beta_type, pos_type, shared, n, transposed):
    from trimkv_b200 import TrimKVCache
    g = torch.Generator(device=DEV).manual_seed(n)
    b, h, d, m, room = 2, 3, 64, 100, 30
    k, v = (torch.randn(b, h, n, d, generator=g, device=DEV).bfloat16() for _ in range(2))
    beta = -torch.rand(b, h, n, generator=g, device=DEV).to(beta_type)
    if transposed:
        beta = beta.transpose(1, 2).contiguous().transpose(1, 2)
    pos = torch.arange(n, device=DEV, dtype=pos_type) + 5
    if not shared:
        pos = pos.expand(b, h, n) + torch.arange(b * h, device=DEV, dtype=pos_type).view(b, h, 1)
    at = pos.expand(b, h, n)
    cache = TrimKVCache(device=DEV)
    cache.update(k, v, beta, pos, 0)
    cache.compress(strategy="alpha", memory_size=m, buffer_size=room)
    cache.check_status()
    score = beta.float() * (n + 1 - at).float()
    keep = score.sort(dim=-1, descending=True, stable=True).indices[..., :m].sort(dim=-1).values if n >= m + room else torch.arange(n, device=DEV).expand(b, h, n)
    assert torch.equal(cache.kv_positions[0].long(), at.long().gather(2, keep))
    assert torch.equal(cache.retention_weights[0], beta.float().gather(2, keep))
    assert torch.equal(cache.key_cache[0], k.gather(2, keep[..., None].expand(-1, -1, -1, d)))
    assert torch.equal(cache.value_cache[0], v.gather(2, keep[..., None].expand(-1, -1, -1, d)))


# on both sides of the lengths where the width changes, in place and in the selection; kept rows that outweigh the keys and that do not
@pytest.mark.gpu
@pytest.mark.parametrize("nseg,n,m", [
    (148, 256, 200), (148, 257, 200), (148, 1024, 900), (148, 1025, 900), (148, 2047, 1500), (148, 2048, 2000), (2, 8191, 4096), (2, 8192, 4096),
    (149, 256, 99), (149, 257, 256), (193, 512, 500), (193, 513, 512), (149, 1024, 1000), (192, 1025, 1024), (193, 1025, 1024), (193, 1025, 300), (296, 1535, 700), (296, 1536, 700),
    (297, 1536, 700), (3, 14337, 5000),
])
def test_widths_agree_where_the_length_decides(nseg, n, m):
    test_widths_agree(nseg, n, m)


# the selection's digits start where the keys first differ and end where a digit's keys all stay: scores that differ in the sign, in one
# bit, nowhere, in a few values, in everything; the fewest and the most kept; the longest segment
@pytest.mark.gpu
@pytest.mark.parametrize("n", [33, 1030, 57000])
@pytest.mark.parametrize("kind", ["equal", "low_bit", "sign", "few", "wide", "narrow", "infinite"])
def test_selection_of_any_scores(n, kind):
    g = torch.Generator(device=DEV).manual_seed(n)
    nseg = 3
    draw = torch.randint(0, 2, (nseg, n), generator=g, device=DEV)
    score = {"equal": lambda: torch.full((nseg, n), -1.5, device=DEV),
             "low_bit": lambda: (draw + 0x3F800000).int().view(torch.float32),
             "sign": lambda: draw * 2.0 - 1.0,
             "few": lambda: -torch.randint(0, 5, (nseg, n), generator=g, device=DEV).float(),
             "wide": lambda: torch.randn(nseg, n, generator=g, device=DEV) * 10.0 ** torch.randint(-30, 30, (nseg, n), generator=g, device=DEV),
             "narrow": lambda: (torch.randint(0, 5000, (nseg, n), generator=g, device=DEV) + 0x3F800000).int().view(torch.float32),
             "infinite": lambda: torch.where(draw == 1, float("-inf"), torch.randn(nseg, n, generator=g, device=DEV))}[kind]()
    pos = torch.full((n,), 6, dtype=torch.int32, device=DEV)                         # q_idx - pos = 1: the score is log beta itself
    for m in sorted({1, 2, n // 2, n - n // 8, n - 1}):
        keep = score.sort(dim=1, descending=True, stable=True).indices[:, :m].sort(dim=1).values
        kept, count = torch.empty(nseg, m, dtype=torch.int32, device=DEV), torch.empty(nseg, dtype=torch.int32, device=DEV)
        status = ops.new_status(DEV)
        ops.evict_select(score, pos, None, n, nseg, 7, m, m, n, kept, count, status)
        assert ops.read_status(status) == 0 and bool((count == m).all())
        assert torch.equal(kept.long(), keep)


# few segments: clusters of 8, 4 and 2 CTAs share a segment's columns, on both sides of the numbers of segments where that changes; rows
# of 64 bytes a slice and fewer, of a width that is no power of two, in 32 bits; uneven lengths, segments that keep everything or nothing
@pytest.mark.gpu
@pytest.mark.parametrize("nseg", [1, 8, 9, 37, 38, 74, 75])
@pytest.mark.parametrize("dim,dtype", [(128, torch.bfloat16), (64, torch.float16), (32, torch.bfloat16), (8, torch.bfloat16), (96, torch.bfloat16),
                                       (128, torch.float32), (256, torch.float32)])
def test_slices_agree(nseg, dim, dtype):
    g = torch.Generator(device=DEV).manual_seed(nseg + dim)
    n, cap = 1111, 1117
    k, v = (torch.randn(nseg * cap, dim, generator=g, device=DEV).to(dtype) for _ in range(2))
    beta, pos = -torch.rand(nseg * cap, generator=g, device=DEV), torch.arange(cap, dtype=torch.int32, device=DEV).repeat(nseg)
    lens = torch.randint(0, n + 1, (nseg,), generator=g, device=DEV).int()
    lens[0] = n
    m = torch.randint(0, n + 1, (nseg,), generator=g, device=DEV).int().clamp(max=lens)
    m[0] = 700
    want = []
    for s in range(nseg):
        at = slice(s * cap, s * cap + int(lens[s]))
        score = beta[at] * (n + 1 - pos[at]).float()
        keep = score.sort(descending=True, stable=True).indices[:int(m[s])].sort().values
        want.append([t[at][keep] for t in (k, v, beta, pos)])
    status, ln, kept = ops.new_status(DEV), lens.clone(), torch.full((nseg, n), -1, dtype=torch.int32, device=DEV)
    ops.evict_ex(k, v, beta, pos, ln, None, nseg, nseg, cap, n + 1, n, m, kept_idx_out=kept, kept_stride=n, status=status)
    assert ops.read_status(status) == 0 and torch.equal(ln, m)
    for s in range(nseg):
        for t, w in zip((k, v, beta, pos), want[s]):
            assert torch.equal(t[s * cap:s * cap + int(m[s])], w)
        if m[s] < lens[s]:
            assert torch.equal(kept[s, :int(m[s])], want[s][3]), s          # a segment's positions count its rows


# ranges of rows in turns, where there are too many segments for clusters (75 and more) and where rows do not divide into slices
@pytest.mark.gpu
@pytest.mark.parametrize("nseg,dim", [(74, 64), (75, 64), (130, 64), (3, 8)])
def test_ranges_of_rows_agree(nseg, dim):
    g = torch.Generator(device=DEV).manual_seed(nseg)
    n, m, cap, ctas = 900, 700, 903, 4
    k, v = (torch.randn(nseg * cap, dim, generator=g, device=DEV).bfloat16() for _ in range(2))
    beta, pos = -torch.rand(nseg * cap, generator=g, device=DEV), torch.arange(cap, dtype=torch.int32, device=DEV).repeat(nseg)
    keep = (beta.view(nseg, cap)[:, :n] * (n + 1 - pos[:n]).float()).sort(dim=1, descending=True, stable=True).indices[:, :m].sort(dim=1).values
    want = [t.view(nseg, cap, -1).gather(1, keep[:, :, None].expand(-1, -1, t.numel() // (nseg * cap))) for t in (k, v, beta, pos)]
    status, ln = ops.new_status(DEV), torch.full((nseg,), n, dtype=torch.int32, device=DEV)
    ops.evict_multi(k, v, beta, pos, ln, None, nseg, nseg, cap, n + 1, m, m, n, ctas, ops.evict_multi_workspace(nseg, m, ctas, torch.device(DEV)), status=status)
    assert ops.read_status(status) == 0 and bool((ln == m).all())
    for t, w in zip((k, v, beta, pos), want):
        assert torch.equal(t.view(nseg, cap, -1)[:, :m], w)


# protected rows are left out of the search unless other rows at infinity, or without a number, take their places; protected rows up to
# and beyond what is kept
@pytest.mark.gpu
@pytest.mark.parametrize("nseg,n", [(3, 1111), (75, 640), (300, 700)])
@pytest.mark.parametrize("kind", ["equal", "wide", "infinite", "no_number", "lowest"])
def test_protected_rows(nseg, n, kind):
    g = torch.Generator(device=DEV).manual_seed(n)
    beta = {"equal": lambda: torch.full((nseg, n), -1.5, device=DEV),
            "wide": lambda: torch.randn(nseg, n, generator=g, device=DEV),
            "infinite": lambda: torch.where(torch.rand(nseg, n, generator=g, device=DEV) < 0.5, float("inf"), -1.0),
            "no_number": lambda: torch.where(torch.rand(nseg, n, generator=g, device=DEV) < 0.3, float("nan"), -1.0),
            "lowest": lambda: torch.where(torch.rand(nseg, n, generator=g, device=DEV) < 0.3, float("-inf"), torch.finfo(torch.float32).min)}[kind]()
    m, dim = n * 3 // 5, 64
    for w in (1, 64, n // 5, m - 1, m, n - 1):
        k, v = (torch.randn(nseg * n, dim, generator=g, device=DEV).bfloat16() for _ in range(2))
        score = beta.double().clone()
        score[:, n - w:] = float("inf")
        score = torch.where(score.isnan(), 1e301, score.clamp(max=1e300))                     # no number: above infinity
        keep = score.sort(dim=1, descending=True, stable=True).indices[:, :m].sort(dim=1).values
        want = [t.view(nseg, n, dim).gather(1, keep[:, :, None].expand(-1, -1, dim)) for t in (k, v)]
        status, ln = ops.new_status(DEV), torch.full((nseg,), n, dtype=torch.int32, device=DEV)
        pos = torch.full((nseg * n,), 6, dtype=torch.int32, device=DEV)                       # the score is log beta itself
        ops.evict_ex(k, v, beta.clone().view(-1), pos, ln, None, nseg, nseg, n, 7, n, None, w, m, m, status=status)
        assert ops.read_status(status) == 0 and bool((ln == m).all())
        for t, x in zip((k, v), want):
            assert torch.equal(t.view(nseg, n, dim)[:, :m], x), w
