"""One token of the SSD layers by a CTA per head and by a CTA per several heads of a group: the same bits, whatever the batch chooses."""
import pytest
import torch

from trimkv_b200 import ops
from trimkv_b200.state_cache import HybridStateCache, RecurrentState

DEV = torch.device("cuda", 0)


def _step(rows, proj, conv, state, weights, out_type, h, n, p, g, taps, start):
    """One step of the given requests from the given rings and states."""
    ch = h * p + 2 * g * n
    cache = HybridStateCache([RecurrentState(h, n, p, taps, ch)], DEV, out_type)
    cache.open(len(rows))
    if start:
        cache.begin([start] * len(rows))
    data = cache.arrays(0)
    batch = cache.begin(None)
    at = batch.slots.long()
    data["conv"][at], data["state"][at] = conv[rows], state[rows]
    out = torch.empty(len(rows), h * p, dtype=out_type, device=DEV)
    ops.ssd_step(proj[rows].contiguous(), data["conv"], data["state"], batch, *weights, out, g)
    return out, data["conv"][at].clone(), data["state"][at].clone()


# heads per group that divide into the CTAs of a group and that do not; one head per CTA in the single requests (and where a row of the
# state has 128 values); fewer rows of the state than threads hold, odd numbers of taps, a request without a past
@pytest.mark.gpu
@pytest.mark.parametrize("requests,h,n,p,g,taps,start", [
    (40, 64, 128, 64, 8, 4, 9), (150, 20, 128, 64, 4, 4, 1), (99, 12, 64, 32, 2, 3, 5), (60, 33, 32, 16, 3, 4, 2), (37, 64, 128, 64, 8, 4, 0),
    (300, 8, 20, 8, 2, 2, 7), (45, 32, 128, 128, 8, 4, 6), (60, 9, 30, 24, 3, 4, 3),
    # just beyond a group per SM, and two: thirds and halves of a group, a head per CTA, groups that stay together
    (20, 48, 128, 64, 8, 4, 4), (49, 28, 64, 32, 4, 4, 2), (75, 14, 64, 64, 2, 4, 5), (40, 48, 64, 64, 8, 4, 5), (100, 40, 64, 32, 4, 4, 3),
    (20, 24, 128, 64, 8, 4, 6), (20, 32, 64, 64, 8, 4, 6)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_heads_of_a_group_in_one_cta(requests, h, n, p, g, taps, start, dtype):
    gen = torch.Generator(device=DEV).manual_seed(requests)
    ch = h * p + 2 * g * n
    proj = torch.randn(requests, h * p + ch + h, generator=gen, device=DEV).to(dtype)
    conv = torch.randn(requests, taps, ch, generator=gen, device=DEV).to(dtype)
    state = torch.randn(requests, h, n, p, generator=gen, device=DEV)
    weights = [torch.randn(ch, taps, generator=gen, device=DEV), torch.randn(ch, generator=gen, device=DEV),
               torch.randn(h, generator=gen, device=DEV) - 3, torch.randn(h, generator=gen, device=DEV), torch.randn(h, generator=gen, device=DEV)]
    args = (proj, conv, state, weights, dtype, h, n, p, g, taps, start)
    together = _step(list(range(requests)), *args)
    for r in (0, requests // 2, requests - 1):
        for a, b in zip(together, _step([r], *args)):
            assert torch.equal(a[r], b[0])
