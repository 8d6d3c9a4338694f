"""GPU: log-sum-exp of the bf16 forward at head size 64 to the digits that its arithmetic has. Every sixteen keys the last
pair's exponentials come from a cubic; the first fourteen rows of a sequence see none of them."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu
D, EXACT_ROWS = 64, 14


@pytest.mark.parametrize("path", ["split", "interleaved", "via_bf16", "dropout"])
@pytest.mark.parametrize("B,H,S", [(5, 3, 4), (4, 2, 8), (3, 3, 14), (2, 3, 40), (2, 2, 300), (16, 12, 1024)])
def test_lse_of_the_first_rows_and_of_the_others(cuda, B, H, S, path):
    BH, scale = B * H, D ** -0.5
    g = torch.Generator(device=cuda).manual_seed(BH * S)
    q, k, v = (torch.empty(BH, S, D, device=cuda).normal_(0.0, 0.5, generator=g).bfloat16() for _ in range(3))
    lse = torch.full((BH, S), float("nan"), device=cuda)
    if path == "via_bf16":
        ws = torch.empty(dad.flash_f32_via_bf16_workspace_bytes(BH, S, D), dtype=torch.uint8, device=cuda)
        dad.gpu_flash_attention_forward_via_bf16(torch.empty(BH, S, D, device=cuda), lse, q.float(), k.float(), v.float(), BH, S, D,
                                                 scale, ws)
    elif path == "interleaved":
        iq, ik, iv = (t.view(B, H, S, D).transpose(1, 2).reshape(B * S, H * D).contiguous() for t in (q, k, v))
        dad.gpu_flash_attention_forward_bf16_interleaved(torch.empty_like(iq), lse, iq, ik, iv, B, H, S, D, scale)
    else:
        drop = {"rate": 0.1, "seed": 3} if path == "dropout" else {}   # (lse is that of the undropped row)
        dad.gpu_flash_attention_forward_bf16(torch.empty_like(q), lse, q, k, v, BH, S, D, scale, **drop)
    assert dad.device_status() == 0
    hidden = torch.triu(torch.ones(S, S, dtype=torch.bool, device=cuda), 1)
    for u0 in range(0, BH, 32):
        s = (q[u0:u0 + 32].double() @ k[u0:u0 + 32].double().transpose(1, 2)) * scale
        error = (lse[u0:u0 + 32].double() - torch.logsumexp(s.masked_fill(hidden, float("-inf")), -1)).abs()
        # A score is 64 products in four instructions, sum of magnitudes (scaled) about 1.3, at most 2.5: eight roundings
        # of 2^-23 of that, 2.4e-6. exp2 2^-22, a result of at most 4 rounded twice: 0.7e-6.
        assert error[:, :EXACT_ROWS].max().item() < 4e-6
        # The cubic is off by 7.9e-4 of a probability at most, and so is then the sum.
        assert error.max().item() < 8e-4
