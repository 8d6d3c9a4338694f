"""GPU: the head-size-128 forward with two query tiles per CTA (csrc/flash_fwd128_sm100.cu): one and two units per item,
odd numbers of tiles and units, ragged ends, several groups of units, under capture, and against the one-tile kernel,
which smaller launches of the same units take."""
import pytest
import torch

from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu
D = 128


def _inputs(cuda, BH, S):
    g = torch.Generator(device=cuda).manual_seed(BH * 10000 + S)
    return [torch.randn(BH, S, D, device=cuda, generator=g).bfloat16() for _ in range(3)]


def _forward(q, k, v):
    out, lse = torch.full_like(q, float("nan")), torch.full(q.shape[:2], float("nan"), device=q.device)
    dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, q.shape[0], q.shape[1], D, D ** -0.5)
    return out, lse


# sequences of one tile (two units an item, the last alone), of two, three, four, five, seven and 16, beyond a group
@pytest.mark.parametrize("BH,S", [(149, 1), (150, 100), (301, 128), (80, 129), (75, 257), (60, 384), (100, 500), (48, 777),
                                  (200, 640), (60, 2040)])
def test_against_float64_and_the_one_tile_kernel(cuda, BH, S):
    q, k, v = _inputs(cuda, BH, S)
    out, lse = _forward(q, k, v)
    assert dad.device_status() == 0
    assert bool(out.isfinite().all()) and bool(lse.isfinite().all())
    for u in {0, 1, BH // 2, BH - 2, BH - 1}:
        s = (q[u].double() @ k[u].double().T) * D ** -0.5
        s = s.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=cuda), 1), float("-inf"))
        # probabilities and results rounded to bf16, 2^-9 of values below 5 each; lse: fp32 sums of at most 2040 terms
        assert (out[u].double() - torch.softmax(s, -1) @ v[u].double()).abs().max().item() < 2e-2
        assert (lse[u].double() - torch.logsumexp(s, -1)).abs().max().item() < 2e-4
    few = slice(BH - 2, BH)   # (two units: one tile per CTA)
    out1, lse1 = _forward(q[few].contiguous(), k[few].contiguous(), v[few].contiguous())
    assert (out[few].float() - out1.float()).abs().max().item() < 2e-2 and (lse[few] - lse1).abs().max().item() < 2e-4


@pytest.mark.parametrize("BH,S", [(160, 128), (64, 1000)])
def test_captured_and_repeated(cuda, BH, S):
    q, k, v = _inputs(cuda, BH, S)
    want, want_lse = _forward(q, k, v)
    out, lse = torch.empty_like(q), torch.empty_like(want_lse)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(3):
                dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, D ** -0.5)
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(20):
        out.fill_(float("nan"))
        lse.fill_(float("nan"))
        graph.replay()
        assert torch.equal(out, want) and torch.equal(lse, want_lse)   # (a row's order of summation is fixed)
    assert dad.device_status() == 0


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_bad_row_stays_with_itself(cuda, value):
    BH, S, unit, at = 80, 600, 33, 400
    q, k, v = _inputs(cuda, BH, S)
    want, want_lse = _forward(q, k, v)
    q[unit, at, 3] = value
    out, lse = _forward(q, k, v)
    assert not out[unit, at].isfinite().any() and not lse[unit, at].isfinite()
    out[unit, at], lse[unit, at] = want[unit, at], want_lse[unit, at]
    assert torch.equal(out, want) and torch.equal(lse, want_lse)
