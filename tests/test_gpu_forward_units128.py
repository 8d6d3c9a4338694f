"""GPU: at head size 128 a unit's forward result is the same bit for bit whatever launch it is part of, although launches
that fill the GPU and those that do not take different kernels: what lets ranks compute shards of a batch."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu
D = 128


def _forward(q, k, v, scale):
    out, lse = torch.full_like(q, float("nan")), torch.full(q.shape[:2], float("nan"), device=q.device)
    dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, q.shape[0], q.shape[1], D, scale)
    return out, lse


# whole launches fill the GPU; shards of 24, 5 and one do not (the last two at 2048 rows: either side of where all launches
# take the same kernel)
@pytest.mark.parametrize("BH,S", [(301, 1), (192, 100), (192, 128), (150, 129), (120, 300), (100, 500), (96, 777), (192, 1024),
                                  (48, 2048), (48, 2049)])
@pytest.mark.parametrize("growth", [0.0, 6.0])   # keys that grow along the sequence: the accumulators are rescaled
def test_shards_equal_the_whole(cuda, BH, S, growth):
    g = torch.Generator(device=cuda).manual_seed(BH * 10000 + S)
    q, k, v = (torch.randn(BH, S, D, device=cuda, generator=g) for _ in range(3))
    k *= torch.linspace(1.0, 1.0 + growth, S, device=cuda)[None, :, None]
    q, k, v = (t.bfloat16() for t in (q, k, v))
    scale = 0.5 if growth else D ** -0.5
    out, lse = _forward(q, k, v, scale)
    assert bool(out.isfinite().all()) and bool(lse.isfinite().all())
    for first, count in ((0, 24), (BH - 24, 24), (17, 5), (BH - 1, 1)):
        part = slice(first, first + count)
        got, got_lse = _forward(q[part].contiguous(), k[part].contiguous(), v[part].contiguous(), scale)
        assert torch.equal(got, out[part]) and torch.equal(got_lse, lse[part]), (first, count)
    assert dad.device_status() == 0
