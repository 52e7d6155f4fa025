"""The projections of the fused one-token step are the library's products of its inputs, bit for bit.

The q/k/v/gate projection feeds the retention gate, whose log betas decide which rows an eviction keeps, and the head-sharded step of the
same model takes the library's product: another order of the sums would let the two keep different rows."""
import pytest
import torch
import torch.nn.functional as F

from trimkv_b200 import TrimKVCache, TrimKVQwen3Config, TrimKVQwen3ForCausalLM, attn, ops
from trimkv_b200.decoder import FusedDecodeStep

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("batch", [1, 8, 32])
def test_products_of_a_step(batch, monkeypatch):
    """Widths of the models as they are used: products of up to 32 rows with 2048 to 6144 columns."""
    cfg = TrimKVQwen3Config(vocab_size=4096, hidden_size=2048, intermediate_size=6144, num_hidden_layers=2, num_attention_heads=16,
                            num_key_value_heads=8, head_dim=128, retention_gate_intermediate_size=128, retention_gate_bias_init=3.0,
                            memory_size=64, buffer_size=16, initializer_range=0.02)
    torch.manual_seed(batch)
    model = TrimKVQwen3ForCausalLM(cfg).to(torch.bfloat16).eval().to(DEV)
    ids = torch.randint(0, cfg.vocab_size, (batch, 41), device=DEV)
    pairs = []                                             # (input, what was made of it), in the order of the step
    with torch.no_grad():
        cache = TrimKVCache(device=DEV)
        model(input_ids=ids[:, :40], past_key_values=cache, logits_to_keep=1)
        step = FusedDecodeStep(model, cache)
        norm, silu, attend, prep = ops.add_rmsnorm, ops.silu_mul, attn.tkv_attention_forward, cache.decode_prep
        src = []

        def made(y):
            pairs.append((src.pop(), y.clone()))

        def add_rmsnorm(x, delta, weight, out, *rest):
            if delta is not None:
                made(delta)
            norm(x, delta, weight, out, *rest)
            src.append(out.clone())

        def silu_mul(gate_up, act, *rest):
            made(gate_up)
            silu(gate_up, act, *rest)
            src.append(act.clone())

        def decode_prep(layer, qkvg, *rest):
            made(qkvg)
            return prep(layer, qkvg, *rest)

        def forward(*args, **kw):
            out = attend(*args, **kw)
            src.append(out[0].view(batch, -1).clone())
            return out

        monkeypatch.setattr(ops, "add_rmsnorm", add_rmsnorm)
        monkeypatch.setattr(ops, "silu_mul", silu_mul)
        monkeypatch.setattr(attn, "tkv_attention_forward", forward)
        monkeypatch.setattr(cache, "decode_prep", decode_prep)
        made(step(ids[:, 40:], torch.tensor([40], device=DEV)))
        monkeypatch.undo()
        weights = [w for layer, w_qkvg, _, w_gu, _ in step.layers
                   for w in (w_qkvg, layer.self_attn.o_proj.weight, w_gu, layer.mlp.down_proj.weight)] + [model.lm_head.weight]
        assert not src and len(pairs) == len(weights) == 9
        for i, ((x, y), w) in enumerate(zip(pairs, weights)):
            assert torch.equal(y, F.linear(x, w)), i
        cache.check_status()
