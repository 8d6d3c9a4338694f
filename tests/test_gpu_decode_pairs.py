"""GPU: clusters that share a head of two sequences (csrc/decode.cu, kPairCluster): how the CTAs are divided between a
long and a short one, an odd number of sequences, ties, sequences that are skipped because their cache is full."""
import pytest
import torch

from dadgpt_b200 import _lib
from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu
FULL = -1


# clusters of eight CTAs with two sequences (40 heads) or one (20), three to five of eight or four with two
@pytest.mark.parametrize("H,max_len,D", [(40, 3000, 128), (20, 3000, 128), (40, 900, 64)])
@pytest.mark.parametrize("lengths", [(2500, 3), (700, 700, 700, 700), (0, 1, 2), (1, 2900, 0, 1400, 1399), (FULL, 40, 800), (5, FULL),
                                     (FULL, FULL, 31), (FULL, FULL)])
def test_uneven_sequences_against_float64(cuda, H, max_len, D, lengths):
    B = len(lengths)
    g = torch.Generator(device=cuda).manual_seed(B * max_len + lengths[0])
    cache = dad.KVCacheBF16(B, H, max_len, D, device=cuda)
    cache.k.normal_(generator=g)
    cache.v.normal_(generator=g)
    at = [max_len if n == FULL else min(n, max_len - 1) for n in lengths]
    cache.lengths.copy_(torch.tensor(at, dtype=torch.int32))
    q, kn, vn = (torch.randn(B, H, D, device=cuda, generator=g).bfloat16() for _ in range(3))
    k_ref, v_ref = cache.k.clone(), cache.v.clone()
    out = torch.full_like(q, 7.0)
    dad.decode_attention_bf16(out, q, kn, vn, cache, D ** -0.5)
    assert dad.device_status() == (-1 if FULL in lengths else 0)
    for b, n in enumerate(at):
        if n == max_len:
            assert bool((out[b] == 7.0).all())
            continue
        k_ref[b, :, n], v_ref[b, :, n] = kn[b], vn[b]
        s = torch.einsum("hd,hld->hl", q[b].double(), k_ref[b, :, :n + 1].double()) * D ** -0.5
        want = torch.einsum("hl,hld->hd", torch.softmax(s, -1), v_ref[b, :, :n + 1].double())
        # fp32 sums, rounded to bf16 once: half a unit of 2^-8 of values below 8
        assert (out[b].double() - want).abs().max().item() < 2e-2
    assert torch.equal(cache.k, k_ref) and torch.equal(cache.v, v_ref)
    assert cache.lengths.tolist() == [n if n == max_len else n + 1 for n in at]


# fp32: clusters of eight (40 heads: two or three sequences; short caches of 32 columns) and of four (the others)
@pytest.mark.parametrize("D,max_len", [(16, 900), (16, 3000), (32, 900), (64, 2000), (128, 900)])
@pytest.mark.parametrize("lengths", [(800, 3), (700, 700, 700, 700), (1, 890, 0, 400, 399), (FULL, 40, 800, 17), (5, FULL)])
def test_uneven_fp32_sequences_against_float64(cuda, D, max_len, lengths):
    lib = _lib.load()
    B, H, scale = len(lengths), 40, D ** -0.5
    g = torch.Generator(device=cuda).manual_seed(B * max_len + D)
    k, v = (torch.randn(B, H, max_len, D, device=cuda, generator=g) for _ in range(2))
    q, kn, vn = (torch.randn(B, H, D, device=cuda, generator=g) for _ in range(3))
    at = [max_len if n == FULL else n for n in lengths]
    lens = torch.tensor(at, dtype=torch.int32, device=cuda)
    ws_bytes = lib.dadattn_decode_workspace_bytes(B, H, D, max_len)
    ws = torch.zeros(ws_bytes, dtype=torch.uint8, device=cuda)
    k_ref, v_ref = k.clone(), v.clone()
    out = torch.full_like(q, 7.0)
    rc = lib.dadattn_decode_f32_batched(out.data_ptr(), q.data_ptr(), kn.data_ptr(), vn.data_ptr(), k.data_ptr(), v.data_ptr(),
                                        lens.data_ptr(), B, H, D, max_len, scale, ws.data_ptr(), ws_bytes,
                                        torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.dadattn_last_error()
    assert dad.device_status() == (-1 if FULL in lengths else 0)
    for b, n in enumerate(at):
        if n == max_len:
            assert bool((out[b] == 7.0).all())
            continue
        k_ref[b, :, n], v_ref[b, :, n] = kn[b], vn[b]
        s = torch.einsum("hd,hld->hl", q[b].double(), k_ref[b, :, :n + 1].double()) * scale
        want = torch.einsum("hl,hld->hd", torch.softmax(s, -1), v_ref[b, :, :n + 1].double())
        # scores: up to 128 products, a few 2^-24 of magnitudes below 10; weights to that, of values below 5
        assert (out[b].double() - want).abs().max().item() < 1e-5
    assert torch.equal(k, k_ref) and torch.equal(v, v_ref)
    assert lens.tolist() == [n if n == max_len else n + 1 for n in at]
