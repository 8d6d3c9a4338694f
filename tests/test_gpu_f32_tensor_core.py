"""GPU: the exact fp32 kernels on the tensor cores (head sizes 16, 32, 64) against float64, at the edges of
their tiles (64 streamed rows, 128 resident rows) and of the rule that gives delta a kernel of its own."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


def _reference(q, k, v, dout, scale, keep=None, rate=0.0):
    q, k, v, dout = (x.double() for x in (q, k, v, dout))
    S = q.shape[1]
    s = (q @ k.transpose(1, 2)) * scale
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - lse[..., None])
    w = torch.ones_like(p) if keep is None else keep.double() / (1 - rate)
    out = (p * w) @ v
    dp = (dout @ v.transpose(1, 2)) * w
    ds = p * (dp - (dout * out).sum(-1, keepdim=True)) * scale
    return out, lse, ds @ k, ds.transpose(1, 2) @ q, (p * w).transpose(1, 2) @ dout


def _run(q, k, v, dout, scale, **drop):
    BH, S, D = q.shape
    out, dq, dk, dv = (torch.full_like(q, float("nan")) for _ in range(4))
    lse, delta = (torch.full((BH, S), float("nan"), device=q.device) for _ in range(2))
    dad.gpu_flash_attention_forward(out, lse, q, k, v, BH, S, D, scale, **drop)
    dad.gpu_flash_attention_backward(dq, dk, dv, delta, dout, out, lse, q, k, v, BH, S, D, scale, **drop)
    assert dad.device_status() == 0
    return out, lse, dq, dk, dv


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("S", [17, 63, 65, 128, 191, 193, 511, 512, 577, 1100])
def test_against_float64(cuda, S, D):
    g = torch.Generator(device=cuda).manual_seed(S * D)
    q, k, v, dout = (torch.randn(2, S, D, device=cuda, generator=g) for _ in range(4))
    got = _run(q, k, v, dout, D ** -0.5)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, _reference(q, k, v, dout, D ** -0.5)):
        assert ((a.double() - b).norm() / b.norm()).item() < 2e-6, name


@pytest.mark.parametrize("offset", [0, 6])   # the draw is word 0, word 2 of its Philox block
@pytest.mark.parametrize("S,D", [(70, 16), (301, 32), (520, 64)])
def test_dropout_draws_the_reference_mask(cuda, S, D, offset):
    g = torch.Generator(device=cuda).manual_seed(S)
    q, k, v, dout = (torch.randn(3, S, D, device=cuda, generator=g) for _ in range(4))
    keep = torch.empty(3 * S * S, dtype=torch.uint8, device=cuda)
    dad.dropout_mask(keep, 0.3, 11, offset, first=5 * S * S)
    got = _run(q, k, v, dout, D ** -0.5, rate=0.3, seed=11, offset=offset, unit0=5)
    want = _reference(q, k, v, dout, D ** -0.5, keep.view(3, S, S), 0.3)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        assert ((a.double() - b).norm() / b.norm()).item() < 2e-6, name


def test_unaligned_tensors_and_repeatability(cuda):
    S, D = 200, 64
    buf = torch.randn(5, 2 * S * D + 1, device=cuda)
    q, k, v, dout = (b[1:].view(2, S, D) for b in buf[:4])
    a = _run(q, k, v, dout, 0.125)
    b = _run(*(x.clone() for x in (q, k, v, dout)), 0.125)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("rate", [0.0, 0.25])
@pytest.mark.parametrize("BH,S,D", [(150, 100, 16), (149, 129, 64), (75, 193, 32), (50, 300, 64), (110, 513, 64), (37, 700, 32)])
def test_several_items_per_cta(cuda, BH, S, D, rate):
    """More tiles than CTAs, ragged, so that a CTA goes from key tiles to query tiles and back."""
    g = torch.Generator(device=cuda).manual_seed(S + D)
    q, k, v, dout = (torch.randn(BH, S, D, device=cuda, generator=g) for _ in range(4))
    keep, drop = None, {}
    if rate:
        drop = {"rate": rate, "seed": 5, "offset": 0, "unit0": 2}
        keep = torch.empty(BH * S * S, dtype=torch.uint8, device=cuda)
        dad.dropout_mask(keep, rate, 5, 0, first=2 * S * S)
        keep = keep.view(BH, S, S)
    got = _run(q, k, v, dout, D ** -0.5, **drop)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, _reference(q, k, v, dout, D ** -0.5, keep, rate)):
        err = (a.double() - b).flatten(1).norm(dim=1) / b.flatten(1).norm(dim=1)
        assert err.max().item() < 3e-6, name
