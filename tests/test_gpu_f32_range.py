"""GPU: the range of the exact fp32 kernels at head sizes 16-64, whose operands are split into bf16 planes:
every finite number, bf16's largest (3.3895e38) or beyond it, and what an infinity leaves behind."""
import pytest
import torch

from tests.test_gpu_f32_tensor_core import _reference, _run

pytestmark = pytest.mark.gpu
FLT_MAX = 3.4028234663852886e38


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("value", [3.3895e38, 3.3953e38, 3.4e38, FLT_MAX, -FLT_MAX, -3.396e38])
def test_values_beyond_the_largest_bf16(cuda, D, value):
    """One key: the output is its V, to the last bit."""
    q = torch.ones(2, 1, D, device=cuda)
    v = torch.full_like(q, value)
    out, lse, dq, dk, dv = _run(q, q, v, torch.zeros_like(q), 0.125)
    assert torch.equal(out, v)


@pytest.mark.parametrize("exponent", [-149, -130, -126, -120, -112, -108, -90])
def test_small_values(cuda, exponent):
    """One key again. Half the spacing of bf16's smallest numbers, 2^-133, is all that may be lost."""
    g = torch.Generator(device=cuda).manual_seed(7)
    q = torch.ones(50, 1, 64, device=cuda)
    v = ((1 + torch.rand(50, 1, 64, device=cuda, generator=g, dtype=torch.float64)) * 2.0 ** exponent).float()
    out, lse, dq, dk, dv = _run(q, q, v, torch.zeros_like(q), 0.125)
    assert (out.double() - v.double()).abs().max().item() <= 2.0 ** -134
    if exponent >= -109:
        assert torch.equal(out, v)


@pytest.mark.parametrize("D", [16, 64])
@pytest.mark.parametrize("S", [65, 300])
def test_products_of_the_largest_numbers(cuda, D, S):
    """K from 3.39e38 up, Q and the scale such that the scores are ordinary numbers."""
    g = torch.Generator(device=cuda).manual_seed(S)
    q, k, v, dout = (torch.randn(2, S, D, device=cuda, generator=g) for _ in range(4))
    q *= 2.0 ** -100
    # dK is of the size of scale q dout = 2^-130 dout. With dout around 1 it is subnormal, and each of its
    # sums then rounds by up to 2^-150 however large it is itself; at 2^20 the relative bound holds.
    dout *= 2.0 ** 20
    k = (k.sign() * (3.39e38 + 1.2e36 * torch.rand(k.shape, device=cuda, generator=g))).contiguous()
    got, want = _run(q, k, v, dout, 2.0 ** -30), _reference(q, k, v, dout, 2.0 ** -30)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        assert a.isfinite().all(), name
        assert ((a.double() - b).norm() / b.norm()).item() < 2e-6, name


@pytest.mark.parametrize("D", [16, 64])
def test_an_infinity_stays_in_its_unit_and_is_seen(cuda, D):
    S, at = 300, 150
    g = torch.Generator(device=cuda).manual_seed(D)
    q, k, v, dout = (torch.randn(3, S, D, device=cuda, generator=g) for _ in range(4))
    clean = _run(q, k, v, dout, 0.125)
    for x in (q, k, v):
        y = x.clone()
        y[1, at, 3] = float("inf")
        got = _run(*(y if t is x else t for t in (q, k, v)), dout, 0.125)
        for a, b in zip(got, clean):
            assert torch.equal(a[[0, 2]], b[[0, 2]])
        rows = [at] if x is q else list(range(at, S))   # the queries that see it
        assert not got[0][1, rows].isfinite().all(-1).any()
        assert torch.equal(got[0][1, :128], clean[0][1, :128])   # query tiles ahead of it are untouched
