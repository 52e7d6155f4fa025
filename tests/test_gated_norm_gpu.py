"""The group norm's forms for 8, 16 and 32 lanes per group and the general one behind them, where a CTA's groups end."""
import numpy as np
import pytest
import torch

from oracle import dafovik_oracle as orc
from tests.test_dafovik_gpu import BF16, DEV, F32, as_held, on_gpu
from trimkv_b200 import ops


# lengths with both vectors of every lane, of some lanes and none of the second; a CTA holds 32, 16 or 8 groups (520: a warp each, in turn)
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("length,held", [(8, 32), (64, 32), (72, 32), (128, 32), (136, 16), (256, 16), (264, 8), (512, 8), (520, 8)])
@pytest.mark.parametrize("groups,over", [(1, -1), (1, 0), (1, 1), (1, 33), (3, 1)])
def test_ends_of_ctas(dtype, length, held, groups, over):
    rng = np.random.default_rng(length + over)
    rows, width = held + over, groups * length                     # groups = 3: a row's groups in two CTAs
    y = as_held(rng.standard_normal((rows, width)) * 10.0 ** rng.integers(-2, 3, (rows, 1)), dtype)
    wide = as_held(rng.standard_normal((rows, width + 24)), dtype)
    z, w = wide[:, 8:8 + width], as_held(rng.standard_normal(width), F32)
    zd, each = on_gpu(wide, dtype)[:, 8:8 + width], y.reshape(rows, groups, length)
    # fp32: a sum of up to 520 squares, a root and four products of 2^-24 each; bf16: those and the rounding of the result
    tol = 2e-6 if dtype is F32 else 2.0 ** -8
    plain = orc.unit_rms(each, 1e-4).reshape(rows, width)

    def near(out, want):
        return (np.abs(out.double().cpu().numpy() - want) <= tol * np.maximum(np.abs(want), 1e-3)).all()
    for gate, weight, first, want in ((zd, w, True, orc.grouped_gated_norm(y, z, w, groups, 1e-4)), (zd, None, False, plain * orc.silu(z)),
                                      (None, w[:length], False, plain * np.tile(w[:length], groups))):
        out = torch.full((rows + 1, width), 7.0, dtype=dtype, device=DEV)
        ops.gated_norm(on_gpu(y, dtype), gate, None if weight is None else on_gpu(weight), out[:rows], groups, 1e-4, gate_first=first)
        assert near(out[:rows], want) and bool((out[rows:] == 7.0).all())
    inplace = on_gpu(y, dtype)
    ops.gated_norm(inplace, zd, None, inplace, groups, 1e-4)
    assert near(inplace, plain * orc.silu(z))
