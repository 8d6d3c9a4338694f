"""GPU: bf16 attention at head size 128 where the CTAs go level by level over groups of units: last groups that are
padded, groups of one unit, groups of thousands."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("BH,S", [(1, 1), (3, 129), (33, 1000), (9, 4096), (2, 20000), (2048, 100), (2049, 100)])
def test_groups_of_units(cuda, BH, S):
    D, scale = 128, 128 ** -0.5
    g = torch.Generator(device=cuda).manual_seed(S + BH)
    q, k, v, dout = (torch.randn(BH, S, D, device=cuda, generator=g).bfloat16() for _ in range(4))
    out, dq, dk, dv = (torch.full_like(q, float("nan")) for _ in range(4))
    lse = torch.full((BH, S), float("nan"), device=cuda)
    ws = torch.full((dad.flash_backward_bf16_workspace_bytes(BH, S, D),), 255, dtype=torch.uint8, device=cuda)
    dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, scale)
    dad.gpu_flash_attention_backward_bf16(dq, dk, dv, ws, dout, out, lse, q, k, v, BH, S, D, scale)
    assert dad.device_status() == 0
    assert all(torch.isfinite(t).all() for t in (out, lse, dq, dk, dv))
    mask = torch.ones(S, S, dtype=torch.bool, device=cuda).triu(1)
    for u in sorted({0, BH // 2, BH - 2, BH - 1} & set(range(BH))):
        a, b, c = (t[u].float().requires_grad_() for t in (q, k, v))
        want = torch.softmax((a @ b.T * scale).masked_fill(mask, float("-inf")), -1) @ c
        want.backward(dout[u].float())
        assert (out[u].float() - want).abs().max().item() < 2e-2
        for got, ref in ((dq[u], a.grad), (dk[u], b.grad), (dv[u], c.grad)):
            assert (got.float() - ref).abs().max().item() < 2e-2 * max(1.0, ref.abs().max().item())
