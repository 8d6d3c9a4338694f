"""GPU: forward over a long sequence with dropout drawn in the kernel. The draws set the softmax warps apart by
more than a tile's arithmetic, so that one may be a tile ahead of another: results must be those of the
reference and the same every time (at head size 128 one barrier for both score buffers let the products start on
half a tile's probabilities)."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu
RATE, SEED = 0.1, 42


def _reference(q, k, v, unit, scale):
    """One unit in float64: its output, its lse, and how much rounding to bf16 (8 significant bits) may move each
    output: every probability by 2^-8 of itself, then the output by 2^-8 of itself."""
    S = q.shape[1]
    mask = torch.empty(S * S, dtype=torch.uint8, device=q.device)
    dad.dropout_mask(mask, RATE, SEED, first=unit * S * S)
    a, b, c = (t[unit].double() for t in (q, k, v))
    s = (a @ b.T * scale).masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    p = torch.softmax(s, -1) * mask.view(S, S) / (1 - RATE)
    out = p @ c
    return out, torch.logsumexp(s, -1), 2.0 ** -8 * (p @ c.abs() + out.abs())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S", [1000, 3080])
def test_long_forward_with_dropout_repeats(S, D):
    BH, scale = 8, D ** -0.5
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.empty(BH, S, D, device="cuda", dtype=torch.bfloat16).normal_(0.0, 0.5, generator=g) for _ in range(3))
    first = None
    for _ in range(20):
        out, lse = torch.empty_like(q), torch.empty(BH, S, device="cuda")
        dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, scale, rate=RATE, seed=SEED)
        assert torch.isfinite(out.float()).all() and torch.isfinite(lse).all()
        if first is None:
            first = out, lse
        assert torch.equal(out, first[0]) and torch.equal(lse, first[1])
    for unit in range(BH):
        want, want_lse, bound = _reference(q, k, v, unit, scale)
        # on top of the roundings: fp32 sums over S terms, and at head size 64 one pair of exponentials in eight
        # comes from a cubic with a relative error of 6e-4, in the numerator and in the sum
        slack = 1e-5 + (6e-4 * 2 ** 8 * bound if D == 64 else 0.0)
        assert ((first[0][unit].double() - want).abs() <= bound + slack).all(), unit
        assert (first[1][unit].double() - want_lse).abs().max().item() <= (1e-3 if D == 64 else 1e-5), unit
    assert dad.device_status() == 0
