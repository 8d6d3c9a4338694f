"""GPU: what a NaN or infinite query row leaves behind in the bf16 kernels. Other rows of the forward, dV of the
keys that the row's query does not see, and other units have to be what they are without it."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


def _steps(B, H, S, D, path, q, k, v, dout, rate):
    """Forward and backward of [B*H,S,D] tensors by the given path: out, lse, dk, dv."""
    BH, scale, dev = B * H, D ** -0.5, q.device
    if path == "via_bf16":
        q, k, v, dout = (t.float() for t in (q, k, v, dout))
        ws = torch.empty(dad.flash_f32_via_bf16_workspace_bytes(BH, S, D), dtype=torch.uint8, device=dev)
    else:
        ws = torch.empty(dad.flash_backward_bf16_workspace_bytes(BH, S, D), dtype=torch.uint8, device=dev)
    if path == "interleaved":
        q, k, v, dout = (t.view(B, H, S, D).transpose(1, 2).reshape(B * S, H * D).contiguous() for t in (q, k, v, dout))
    out, lse = torch.empty_like(q), torch.empty(BH, S, device=dev)
    dq, dk, dv = (torch.empty_like(q) for _ in range(3))
    if path == "via_bf16":
        dad.gpu_flash_attention_forward_via_bf16(out, lse, q, k, v, BH, S, D, scale, ws)
        dad.gpu_flash_attention_backward_via_bf16(dq, dk, dv, dout, out, lse, q, k, v, BH, S, D, scale, ws)
    elif path == "interleaved":
        dad.gpu_flash_attention_forward_bf16_interleaved(out, lse, q, k, v, B, H, S, D, scale)
        dad.gpu_flash_attention_backward_bf16_interleaved(dq, dk, dv, ws, dout, out, lse, q, k, v, B, H, S, D, scale)
    else:
        drop = {"rate": rate, "seed": 5} if rate else {}
        if path == "masked":
            drop["mask_bits"] = dad.dropout_mask_bits(BH, S, rate, 5)
        dad.set_backward_deterministic(path == "two_kernel")
        try:
            dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, scale, **drop)
            dad.gpu_flash_attention_backward_bf16(dq, dk, dv, ws, dout, out, lse, q, k, v, BH, S, D, scale, **drop)
        finally:
            dad.set_backward_deterministic(False)
    if path == "interleaved":
        out, dk, dv = (t.view(B, S, H, D).transpose(1, 2).reshape(BH, S, D) for t in (out, dk, dv))
    assert dad.device_status() == 0
    return out, lse, dk, dv


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("D,path,rate", [(64, "single", 0.0), (64, "single", 0.1), (64, "masked", 0.1), (64, "interleaved", 0.0),
                                         (64, "via_bf16", 0.0), (64, "two_kernel", 0.0), (128, "single", 0.0),
                                         (128, "single", 0.1), (128, "via_bf16", 0.0), (128, "two_kernel", 0.0)])
@pytest.mark.parametrize("at", [130, 200, 299])   # tile 128-255 of 300 rows, and the last row
def test_a_bad_query_row_stays_with_the_keys_it_sees(cuda, D, path, rate, value, at):
    B, H, S, unit = 2, 2, 300, 1
    g = torch.Generator(device=cuda).manual_seed(D + at)
    q, k, v, dout = (torch.randn(B * H, S, D, device=cuda, generator=g).to(torch.bfloat16) for _ in range(4))
    want = _steps(B, H, S, D, path, q, k, v, dout, rate)
    bad = q.clone()
    bad[unit, at, 3] = value
    got = _steps(B, H, S, D, path, bad, k, v, dout, rate)
    others = [u for u in range(B * H) if u != unit]
    for name, a, b in zip(("out", "lse", "dk", "dv"), got, want):
        assert torch.equal(a[others], b[others]), name
    rows = [r for r in range(S) if r != at]
    assert not got[0][unit, at].isfinite().any()
    assert torch.equal(got[0][unit, rows], want[0][unit, rows])
    assert torch.equal(got[1][unit, rows], want[1][unit, rows])
    # every sum that a masked pair takes part in gets a zero from it
    assert torch.equal(got[3][unit, at + 1:], want[3][unit, at + 1:])
    # dK of the tile's later keys may be lost (0 x NaN), as the interface says; further tiles may not
    after = (at // 128 + 1) * 128
    assert torch.equal(got[2][unit, after:], want[2][unit, after:])
