"""GPU: bf16 forward and backward on sequences of one tile, where the forward gives the two tiles of a work item
to two different (batch, head) units: even and odd numbers of units, one and several items per CTA."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [0, 3])   # 0: heads split, 3: interleaved activations
@pytest.mark.parametrize("BH", [1, 2, 3, 147, 300, 903])
@pytest.mark.parametrize("S", [1, 77, 128])
def test_one_tile_units(cuda, S, BH, heads):
    if heads and BH % heads:
        pytest.skip("whole batch entries only")
    D, scale = 64, 0.125
    g = torch.Generator(device=cuda).manual_seed(S * BH)
    q, k, v = (torch.randn(BH, S, D, device=cuda, generator=g).bfloat16() for _ in range(3))
    out = torch.full_like(q, float("nan"))
    lse = torch.full((BH, S), float("nan"), device=cuda)
    if heads:
        def inter(x):
            return x.view(BH // heads, heads, S, D).transpose(1, 2).reshape(BH // heads * S, heads * D).contiguous()
        got = inter(out)
        dad.gpu_flash_attention_forward_bf16_interleaved(got, lse, inter(q), inter(k), inter(v), BH // heads, heads, S, D,
                                                         scale)
        out = got.view(BH // heads, S, heads, D).transpose(1, 2).reshape(BH, S, D)
    else:
        dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, scale)
    s = (q.float() @ k.float().transpose(1, 2)) * scale
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=cuda).tril(), float("-inf"))
    assert (lse - torch.logsumexp(s, -1)).abs().max().item() < 1e-2
    assert (out.float() - torch.softmax(s, -1) @ v.float()).abs().max().item() < 2e-2
    assert dad.device_status() == 0
