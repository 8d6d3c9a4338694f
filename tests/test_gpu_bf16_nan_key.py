"""GPU: a NaN in a key row of the bf16 forward reaches the result and the log-sum-exp of every row that sees the key,
whichever unit its exponential comes from, and no other."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


# (pairs of columns 16 apart take the same instructions; 60 units of 300 rows at head size 128 fill the GPU, 4 do not)
@pytest.mark.parametrize("D,BH", [(64, 4), (128, 4), (128, 60)])
@pytest.mark.parametrize("first", [0, 16, 128, 272])
def test_a_bad_key_is_seen_by_the_rows_that_see_it(cuda, D, BH, first):
    S, scale, unit = 300, D ** -0.5, 1
    g = torch.Generator(device=cuda).manual_seed(D + first)
    q, k, v = (torch.randn(BH, S, D, device=cuda, generator=g).bfloat16() for _ in range(3))

    def forward(keys):
        out, lse = torch.empty_like(q), torch.empty(BH, S, device=cuda)
        dad.gpu_flash_attention_forward_bf16(out, lse, q, keys, v, BH, S, D, scale)
        return out, lse

    want, want_lse = forward(k)
    for at in range(first, first + 16):
        bad = k.clone()
        bad[unit, at, 5] = float("nan")
        out, lse = forward(bad)
        assert bool(out[unit, at:].isnan().all()) and bool(lse[unit, at:].isnan().all()), at
        out[unit, at:], lse[unit, at:] = want[unit, at:], want_lse[unit, at:]
        assert torch.equal(out, want) and torch.equal(lse, want_lse), at
    assert dad.device_status() == 0
