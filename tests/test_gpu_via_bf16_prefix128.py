"""GPU: at head size 128 the fp32-tensor entry point on bf16 arithmetic sums each half of a row by itself at every length,
as the bf16 entry point does beyond 2048 rows: a sequence's results are those of the longer one that it begins, bit for
bit (lengths of whole warps: rows that share one are rescaled together)."""
import pytest
import torch

import dadgpt_b200 as dad
from dadgpt_b200.attention import device_status, flash_f32_via_bf16_workspace_bytes

pytestmark = pytest.mark.gpu
D, LONG = 128, 2080


@pytest.mark.parametrize("BH", [3, 192])
@pytest.mark.parametrize("S", [32, 128, 160, 800, 2048])
def test_results_are_those_of_the_longer_sequence(cuda, BH, S):
    scale = D ** -0.5
    g = torch.Generator(device=cuda).manual_seed(BH + S)
    long = [torch.randn(BH, LONG, D, device=cuda, generator=g) for _ in range(3)]
    q, k, v = (t[:, :S].contiguous() for t in long)
    out, lse = torch.full_like(q, float("nan")), torch.full((BH, S), float("nan"), device=cuda)
    ws = torch.empty(flash_f32_via_bf16_workspace_bytes(BH, S, D), dtype=torch.uint8, device=cuda)
    dad.gpu_flash_attention_forward_via_bf16(out, lse, q, k, v, BH, S, D, scale, ws)
    bq, bk, bv = (t.bfloat16() for t in long)
    want, want_lse = torch.empty_like(bq), torch.empty(BH, LONG, device=cuda)
    dad.gpu_flash_attention_forward_bf16(want, want_lse, bq, bk, bv, BH, LONG, D, scale)
    assert torch.equal(out, want[:, :S].float()) and torch.equal(lse, want_lse[:, :S])
    assert device_status() == 0
