"""GPU: forward at head size 128 over a long sequence with dropout. The draws set the softmax warps apart by
more than a tile's arithmetic, so that one may be a tile ahead of another: results must be finite and the same
every time (one barrier for both score buffers let the products start on half a tile's probabilities)."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1000, 3080])
def test_long_forward_with_dropout_repeats(S):
    BH, D = 8, 128
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.empty(BH, S, D, device="cuda", dtype=torch.bfloat16).normal_(0.0, 0.5, generator=g) for _ in range(3))
    first = None
    for _ in range(20):
        out, lse = torch.empty_like(q), torch.empty(BH, S, device="cuda")
        dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, D ** -0.5, rate=0.1, seed=42)
        assert torch.isfinite(out.float()).all() and torch.isfinite(lse).all()
        if first is None:
            first = out, lse
        assert torch.equal(out, first[0]) and torch.equal(lse, first[1])
