"""GPU: every way the decode kernel deals out its (sequence, head) pairs: clusters of 2, 4 and 8 CTAs, one
CTA each, persistent CTAs with and without the ranking, more sequences than lengths are copied for."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,max_len,D", [(1, 3, 9000, 64), (2, 5, 4100, 128), (7, 12, 3000, 128), (20, 12, 3000, 64),
                                           (3, 4, 40, 64), (50, 20, 90, 64), (128, 12, 200, 128), (300, 3, 70, 64)])
def test_steps_against_float64(cuda, B, H, max_len, D):
    g = torch.Generator(device=cuda).manual_seed(B * max_len)
    cache = dad.KVCacheBF16(B, H, max_len, D, device=cuda)
    cache.k.normal_(generator=g)
    cache.v.normal_(generator=g)
    lengths = torch.randint(0, max_len - 3, (B,), generator=g, device=cuda, dtype=torch.int32)
    lengths[0], lengths[-1] = max_len - 3, 0
    cache.lengths.copy_(lengths)
    k_ref, v_ref = cache.k.clone(), cache.v.clone()
    rows = torch.arange(max_len, device=cuda)
    for step in range(3):   # the third fills the longest sequence to the last row
        q, kn, vn = (torch.randn(B, H, D, device=cuda, generator=g).bfloat16() for _ in range(3))
        out = torch.full_like(q, float("nan"))
        dad.decode_attention_bf16(out, q, kn, vn, cache, D ** -0.5)
        b = torch.arange(B, device=cuda)
        at = (lengths + step).long()
        k_ref[b, :, at], v_ref[b, :, at] = kn, vn
        s = torch.einsum("bhd,bhld->bhl", q.float(), k_ref.float()) * D ** -0.5
        s = s.masked_fill(rows[None, None] > at[:, None, None], float("-inf"))
        want = torch.einsum("bhl,bhld->bhd", torch.softmax(s, -1), v_ref.float())
        assert (out.float() - want).abs().max().item() < 2e-2
        assert torch.equal(cache.k, k_ref) and torch.equal(cache.v, v_ref)
        assert torch.equal(cache.lengths, lengths + step + 1)
    assert dad.device_status() == 0


@pytest.mark.parametrize("B,H", [(5, 3), (100, 12)])
def test_full_sequences_are_skipped_and_reported(cuda, B, H):
    max_len, D = 33, 64
    cache = dad.KVCacheBF16(B, H, max_len, D, device=cuda)
    cache.lengths[1] = max_len
    x = torch.randn(B, H, D, device=cuda).bfloat16()
    out = torch.full_like(x, 7.0)
    dad.decode_attention_bf16(out, x, x, x, cache, 0.125)
    assert dad.device_status() == -1
    assert bool((out[1] == 7.0).all()) and cache.lengths[1].item() == max_len
    keep = [i for i in range(B) if i != 1]
    assert torch.equal(out[keep], x[keep]) and bool((cache.lengths[keep] == 1).all())
