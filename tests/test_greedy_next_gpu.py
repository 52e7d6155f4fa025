"""The next token of every row and the step's position in one kernel."""
import pytest
import torch

from trimkv_b200 import ops

DEV = "cuda"


# whole vectors and single elements (odd sizes, rows that do not start on 16 bytes), less and more than a round of a CTA
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab,shift", [(1, 0), (7, 0), (8, 0), (1000, 0), (1000, 3), (32768, 0), (50257, 0), (8 * 4096 + 8, 0)])
def test_same_as_argmax(vocab, shift, dtype):
    g = torch.Generator(device=DEV).manual_seed(vocab)
    rows = 6
    z = torch.randn(rows, vocab + 16, generator=g, device=DEV).to(dtype)[:, shift:shift + vocab]
    z[1] = z[1].clamp(max=0.0)                  # many equals: the first counts
    z[2] = float("-inf")
    z[3, vocab // 2:] = float("nan")
    z[4] = -0.0
    z[4, vocab // 3] = 0.0
    z[5, vocab - 1] = float("inf")
    nxt, ids, pos = torch.full((rows, 1), -1, device=DEV), torch.full((rows, 1), -1, device=DEV), torch.tensor([41], device=DEV)
    assert ops.greedy_next(z, nxt, ids, pos)
    want = z.float().cpu().argmax(-1, keepdim=True)
    assert torch.equal(nxt.cpu(), want) and torch.equal(ids.cpu(), want) and pos.item() == 42


@pytest.mark.gpu
def test_logits_it_leaves_alone():
    nxt = torch.zeros(2, 1, dtype=torch.int64, device=DEV)
    pos = torch.zeros(1, dtype=torch.int64, device=DEV)
    z = torch.zeros(2, 64, device=DEV)
    for bad in (z.half(), z.double(), z[None], z.t()[:, :2], z[:0], z.cpu()):
        assert not ops.greedy_next(bad, nxt, nxt, pos)
    assert not ops.greedy_next(z, nxt.int(), nxt, pos) and pos.item() == 0


@pytest.mark.gpu
def test_buffers_of_another_size_are_left_alone():
    """The kernel writes an id per row and one position: fewer or more are for the general path, which raises or broadcasts."""
    z = torch.zeros(3, 64, device=DEV)

    def ints(*shape):
        return torch.full(shape, 9, dtype=torch.int64, device=DEV)
    for sizes in ((2, 3, 1), (3, 2, 1), (4, 3, 1), (3, 4, 1), (0, 3, 1), (3, 3, 2), (3, 3, 0)):
        held = [ints(n) for n in sizes]
        assert not ops.greedy_next(z, *held) and all(bool((t == 9).all()) for t in held)
    held = ints(3, 1), ints(3), ints()
    assert ops.greedy_next(z, *held) and held[0].flatten().tolist() == held[1].tolist() == [0, 0, 0] and held[2].item() == 10


@pytest.mark.gpu
@pytest.mark.parametrize("rows,vocab,taken", [(1, 151936, True), (1, 154000, True), (1, 154001, False), (8, 256000, False), (32, 256000, True)])
def test_large_vocabularies_of_few_rows_are_left_alone(rows, vocab, taken):
    z = torch.randn(rows, vocab, generator=torch.Generator(device=DEV).manual_seed(rows), device=DEV).bfloat16()
    nxt, ids, pos = (torch.zeros(*shape, dtype=torch.int64, device=DEV) for shape in ((rows, 1), (rows, 1), (1,)))
    assert ops.greedy_next(z, nxt, ids, pos) == taken
    if taken:
        want = z.float().cpu().argmax(-1, keepdim=True)
        assert torch.equal(nxt.cpu(), want) and torch.equal(ids.cpu(), want) and pos.item() == 1
