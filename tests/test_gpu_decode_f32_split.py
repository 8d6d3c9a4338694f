"""GPU: one fp32 sequence's rows shared by 1, 2, 4 and 8 CTAs, on both sides of each line."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,D", [(3, 16), (8, 32), (12, 64), (24, 128)])
@pytest.mark.parametrize("kb", [64, 128, 256, 700])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_decode_against_float64(cuda, H, D, kb, more):
    """pos + 1 rows, of which 64 KB of K and V are one CTA's share. 1e-5: fp32 sums, as in the oracle tests."""
    pos = kb * 1024 // (8 * D) + more - 1
    g = torch.Generator(device=cuda).manual_seed(pos)
    k, v = (torch.randn(H, pos + 4, D, device=cuda, generator=g) for _ in range(2))
    q, kn, vn = (torch.randn(H, D, device=cuda, generator=g) for _ in range(3))
    out = torch.full((H, D), float("nan"), device=cuda)
    kr, vr = k.double()[:, :pos + 1].clone(), v.double()[:, :pos + 1].clone()
    kr[:, pos], vr[:, pos] = kn.double(), vn.double()
    dad.decode_attention_f32(out.view(-1), q.view(-1), kn.view(-1), vn.view(-1), k, v, pos, D ** -0.5)
    p = torch.softmax(torch.einsum("hd,hld->hl", q.double(), kr) * D ** -0.5, -1)
    assert (out - torch.einsum("hl,hld->hd", p, vr)).abs().max().item() < 1e-5
    assert torch.equal(k[:, pos], kn) and torch.equal(v[:, pos], vn)
    assert dad.device_status() == 0
