"""Selections whose keys come near the shared memory that a launch gets unasked: 48 KB less what the kernel itself declares.

Each list of lengths runs in a process of its own and ascends, since the first longer segment would raise the limit for the shorter ones."""
import os
import subprocess
import sys

import pytest
import torch

DEV = "cuda"
LENGTHS = (11000, 11226, 11227, 12000, 12288, 12289)


def _check(kind, nseg, dim, ctas):
    from trimkv_b200 import ops
    for n in LENGTHS:
        g = torch.Generator(device=DEV).manual_seed(n)
        m, cap = n - 300, n
        beta, pos = -torch.rand(nseg, cap, generator=g, device=DEV), torch.arange(cap, dtype=torch.int32, device=DEV)
        keep = (beta * (n + 1 - pos).float()).sort(dim=1, descending=True, stable=True).indices[:, :m].sort(dim=1).values
        status = ops.new_status(DEV)
        if kind == "select":
            kept, count = torch.empty(nseg, m, dtype=torch.int32, device=DEV), torch.empty(nseg, dtype=torch.int32, device=DEV)
            ops.evict_select(beta, pos, None, n, nseg, n + 1, m, m, n, kept, count, status)
            assert torch.equal(kept.long(), keep) and bool((count == m).all()), n
        else:
            k, v = (torch.randn(nseg * cap, dim, generator=g, device=DEV, dtype=torch.bfloat16) for _ in range(2))
            want = [t.view(nseg, cap, dim).gather(1, keep[:, :, None].expand(-1, -1, dim)) for t in (k, v)]
            beta, pos = beta.view(-1), pos.repeat(nseg)
            ln = torch.full((nseg,), n, dtype=torch.int32, device=DEV)
            if ctas > 1:
                ops.evict_multi(k, v, beta, pos, ln, None, nseg, nseg, cap, n + 1, m, m, n, ctas,
                                ops.evict_multi_workspace(nseg, m, ctas, torch.device(DEV)), status=status)
            else:
                ops.evict(k, v, beta, pos, ln, None, nseg, nseg, cap, n + 1, m, m, n, status=status)
            assert bool((ln == m).all()), n
            for t, w in zip((k, v), want):
                assert torch.equal(t.view(nseg, cap, dim)[:, :m], w), n
            assert torch.equal(pos.view(nseg, cap)[:, :m].long(), keep), n
        assert ops.read_status(status) == 0, n


# CTAs of 1024 and 512 threads; clusters of 8, 4 and 2 and no cluster; the selection ahead of several CTAs per segment
@pytest.mark.gpu
@pytest.mark.parametrize("kind,nseg,dim,ctas", [("select", 2, 0, 1), ("select", 150, 0, 1), ("select", 300, 0, 1), ("evict", 1, 128, 1), ("evict", 9, 128, 1),
                                                ("evict", 38, 64, 1), ("evict", 75, 64, 1), ("evict", 149, 32, 1), ("evict", 300, 32, 1), ("evict", 75, 64, 2)])
def test_lengths_at_the_limit(kind, nseg, dim, ctas):
    at = os.path.dirname(os.path.abspath(__file__))
    code = f"import sys; sys.path[:0] = [{os.path.dirname(at)!r}, {at!r}]; import test_evict_lengths_gpu as t; t._check({kind!r}, {nseg}, {dim}, {ctas})"
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
