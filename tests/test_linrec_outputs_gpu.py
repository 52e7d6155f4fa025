"""Outputs of the tcgen05 recurrence (csrc/tkv_linrec_tc.cu): a whole chunk leaves as one copy of a tile, a part of a chunk row by row."""
import pytest
import torch

from trimkv_b200 import ops
from trimkv_b200.state_cache import HybridStateCache, RecurrentState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [64, 72, 136])
def test_chunks_whole_and_in_part_stay_within_their_request(p):
    """Requests that end on, before and after a chunk's end give the bits that each gives after the first, and nothing beyond their rows."""
    lens, heads, n = [256, 128, 129, 127, 1, 384], 2, 128
    g = torch.Generator(device="cuda").manual_seed(p)
    T = sum(lens)
    q, k = (torch.randn(T, heads * n, generator=g, device="cuda").bfloat16() * n ** -0.5 for _ in range(2))
    v = torch.randn(T, heads * p, generator=g, device="cuda").bfloat16()
    decay, scale = -torch.rand(T, heads, generator=g, device="cuda") * 0.1, torch.rand(T, heads, generator=g, device="cuda")
    skip = torch.rand(heads, generator=g, device="cuda")

    def run(lens, rows):
        cache = HybridStateCache([RecurrentState(heads, n, p)], torch.device("cuda"), torch.bfloat16)
        cache.open(len(lens))
        out = torch.full((sum(lens) + 128, heads * p), 7.0, dtype=torch.bfloat16, device="cuda")     # rows beyond the last request
        ops.linrec(q[rows], k[rows], v[rows], cache.arrays(0)["state"], cache.begin(list(lens)), out[:sum(lens)], heads, log_decay=decay[rows],
                   v_scale=scale[rows], skip=skip)
        assert bool((out[sum(lens):] == 7.0).all())
        return out[:sum(lens)]

    packed, at = run(lens, torch.arange(T)), 0
    for L in lens:
        after = run([lens[0], L], torch.cat([torch.arange(lens[0]), torch.arange(at, at + L)]))
        assert torch.equal(packed[at:at + L], after[lens[0]:]), L
        at += L
