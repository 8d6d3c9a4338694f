"""GPU: the library's kernels start while the kernel ahead of them in the stream drains; none of them may
touch what that kernel still reads or writes."""
import pytest
import torch

from dadgpt_b200 import attention as dad
from tests import kernel_ahead

pytestmark = pytest.mark.gpu

NAN = 0x7fc00000


@pytest.mark.parametrize("path,D", [("split", 64), ("interleaved", 64), ("split", 128), ("via_bf16", 64)])
def test_backward_workspace_may_be_the_bytes_of_a_call_before(cuda, path, D):
    """The kernel ahead writes all over the bytes that the backward takes as workspace (in an arena: the
    results of an earlier call), late. What the backward clears, it has to clear after that."""
    B, H, S = 2, 2, 300
    BH, scale = B * H, D ** -0.5
    shape = (B * S, H * D) if path == "interleaved" else (BH, S, D)
    g = torch.Generator(device=cuda).manual_seed(D)
    dtype = torch.float32 if path == "via_bf16" else torch.bfloat16
    q, k, v, do = (torch.randn(shape, device=cuda, generator=g).to(dtype) for _ in range(4))
    out, lse = torch.empty_like(q), torch.empty(BH, S, device=cuda)
    nbytes = (dad.flash_f32_via_bf16_workspace_bytes if path == "via_bf16"
              else dad.flash_backward_bf16_workspace_bytes)(BH, S, D)
    ws = torch.zeros(nbytes // 4, dtype=torch.float32, device=cuda)
    grads = [torch.empty_like(q) for _ in range(3)]

    def backward():
        if path == "via_bf16":
            dad.gpu_flash_attention_backward_via_bf16(*grads, do, out, lse, q, k, v, BH, S, D, scale, ws)
        elif path == "interleaved":
            dad.gpu_flash_attention_backward_bf16_interleaved(*grads, ws, do, out, lse, q, k, v, B, H, S, D, scale)
        else:
            dad.gpu_flash_attention_backward_bf16(*grads, ws, do, out, lse, q, k, v, BH, S, D, scale)

    if path == "via_bf16":
        dad.gpu_flash_attention_forward_via_bf16(out, lse, q, k, v, BH, S, D, scale, ws)
    elif path == "interleaved":
        dad.gpu_flash_attention_forward_bf16_interleaved(out, lse, q, k, v, B, H, S, D, scale)
    else:
        dad.gpu_flash_attention_forward_bf16(out, lse, q, k, v, BH, S, D, scale)
    backward()
    torch.cuda.synchronize()
    want = [x.clone() for x in grads]
    for x in grads:
        x.fill_(float("nan"))
    kernel_ahead.launch(ws, value=NAN)   # (loads its module: outside the pair that is tested)
    torch.cuda.synchronize()
    kernel_ahead.launch(ws, value=NAN)
    backward()
    assert dad.device_status() == 0
    for got, ref, name in zip(grads, want, ("dq", "dk", "dv")):
        # dK and dV are summed in a fixed order; dQ in the order of arrival, rounded to bf16 (2^-8) at most
        if name == "dq":
            assert (got.float() - ref.float()).norm() <= 1e-2 * ref.float().norm(), name
        else:
            assert torch.equal(got, ref), name


@pytest.fixture
def early_start():
    dad.set_decode_early_start(True)
    yield
    dad.set_decode_early_start(False)


def _cache(B, H, max_len, D, g):
    cache = dad.KVCacheBF16(B, H, max_len, D)
    cache.k.normal_(generator=g)
    cache.v.normal_(generator=g)
    cache.lengths.copy_(torch.randint(0, max_len - 8, (B,), generator=g, device="cuda", dtype=torch.int32))
    return cache


# clusters, one CTA per pair, persistent CTAs, more sequences than lengths are copied for
@pytest.mark.parametrize("B,H,max_len", [(2, 3, 4000), (3, 4, 60), (64, 12, 300), (300, 3, 60)])
def test_decode_with_early_start_leaves_the_lengths_to_the_kernel_ahead(cuda, early_start, B, H, max_len):
    """The kernel ahead may read the lengths (positions of the tokens): it sees them as they were."""
    g = torch.Generator(device=cuda).manual_seed(B)
    cache = _cache(B, H, max_len, 64, g)
    x = torch.randn(B, H, 64, device=cuda, generator=g).bfloat16()
    out, seen = torch.empty_like(x), torch.empty_like(cache.lengths)
    kernel_ahead.launch(seen, src=cache.lengths)
    before = cache.lengths.clone()
    torch.cuda.synchronize()
    kernel_ahead.launch(seen.fill_(-1), src=cache.lengths)
    dad.decode_attention_bf16(out, x, x, x, cache, 0.125)
    assert dad.device_status() == 0
    assert torch.equal(seen, before) and torch.equal(cache.lengths, before + 1)


def test_decode_with_early_start_overlaps_the_call_ahead_and_no_other(cuda, early_start):
    """Two layers' caches in turn, all calls early: the call on a cache may start beside the other
    cache's call, but not beside the one before it on its own cache, whose rows and lengths it needs.
    The kernel ahead of them all holds everything up until the last call is in the stream."""
    B, H, D, steps = 1, 4, 64, 4
    g = torch.Generator(device=cuda).manual_seed(3)
    caches = [_cache(B, H, 60, D, g) for _ in range(2)]
    again = [_cache(B, H, 60, D, g) for _ in range(2)]
    for c, a in zip(caches, again):
        for name in ("k", "v", "lengths"):
            getattr(a, name).copy_(getattr(c, name))
    x = torch.randn(3, steps, 2, B, H, D, device=cuda, generator=g).bfloat16()
    out, want = torch.empty_like(x[0]), torch.empty_like(x[0])
    dummy = torch.zeros(4, device=cuda)
    kernel_ahead.launch(dummy)
    torch.cuda.synchronize()
    kernel_ahead.launch(dummy, pause=2000)
    for i in range(steps):
        for layer, c in enumerate(caches):
            dad.decode_attention_bf16(out[i, layer], *x[:, i, layer], c, 0.125)
    assert dad.device_status() == 0
    dad.set_decode_early_start(False)
    for i in range(steps):
        for layer, c in enumerate(again):
            dad.decode_attention_bf16(want[i, layer], *x[:, i, layer], c, 0.125)
    assert dad.device_status() == 0
    assert torch.equal(out, want)
    for c, a in zip(caches, again):
        assert torch.equal(c.lengths, a.lengths) and torch.equal(c.k, a.k) and torch.equal(c.v, a.v)
