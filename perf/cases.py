"""The attention work that users of this library have it do, as cases whose speed is followed.

Kinds of case (``kind``):
  train     forward + backward over one layer's attention, a training step's share
  forward   forward alone: prompt ingestion (prefill) and evaluation
  decode    one generated token per sequence, through the layers of a model, against KV caches

``dtype`` of train / forward: "f32" is the exact fp32 path (the drop-in default), "bf16" the
tensor-core path, "via_bf16" fp32 tensors with tensor-core arithmetic (what the drop-in does at
training precision). ``rate`` is the attention dropout; ``layout`` "split" is [B*H, S, D],
"interleaved" the activations as the projections leave them, [B*S, H*D].

Tensors are i.i.d. normal values: activations after layer norm and a projection are close to that.
Buffers for results, workspaces and caches are made once, as a model's arena does.
"""
from __future__ import annotations

import torch

from dadgpt_b200 import attention as dad

TORCH_DTYPE = {"f32": torch.float32, "via_bf16": torch.float32, "bf16": torch.bfloat16}


def _attention(name, kind, dtype, B, H, S, D, rate=0.0, layout="split"):
    c = {"kind": kind, "dtype": dtype, "B": B, "H": H, "S": S, "D": D, "rate": rate, "layout": layout}
    return {"name": name, **c} if name else c


def _decode(name, dtype, layers, B, H, D, max_len, longest, graph):
    c = {"kind": "decode", "dtype": dtype, "layers": layers, "B": B, "H": H, "D": D, "max_len": max_len,
         "longest": longest, "graph": graph}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the tiny preset in exact fp32: smoke tests, gradient checks, CPU-comparable runs
        _attention("train_f32_tiny", "train", "f32", 4, 4, 64, 16),
        # small model with its default attention dropout, ragged length, exact fp32
        _attention("train_f32_dropout_D32", "train", "f32", 4, 8, 301, 32, rate=0.1),
        # GPT-2 124M at full context, batch 4, on the exact fp32 drop-in
        _attention("train_f32_gpt2_b4", "train", "f32", 4, 12, 1024, 64),
        # the same model behind the same fp32 interface at bf16 arithmetic (the training default)
        _attention("train_via_bf16_gpt2_b4", "train", "via_bf16", 4, 12, 1024, 64),
        # GPT-2 124M, batch 16: the benchmark's headline shape
        _attention("train_bf16_gpt2_b16", "train", "bf16", 16, 12, 1024, 64),
        # and with the default training dropout, the mask drawn once per step
        _attention("train_bf16_gpt2_b16_dropout", "train", "bf16", 16, 12, 1024, 64, rate=0.1),
        # a last, shorter batch of a corpus, on activations whose heads were never split
        _attention("train_bf16_ragged_inter", "train", "bf16", 6, 12, 777, 64, layout="interleaved"),
        # long context, head size 128: the benchmark's largest
        _attention("train_bf16_large", "train", "bf16", 8, 24, 8192, 128),
        # a batch of short prompts before generation
        _attention("forward_bf16_T128", "forward", "bf16", 16, 12, 128, 64),
        # DadGPT's own generation loop: one sequence, fp32 caches, direct calls, 12 layers
        _decode("decode_f32_one", "f32", 12, 1, 12, 64, 1024, 700, graph=False),
        # serving, 64 sequences of mixed length, a CUDA graph per token step
        _decode("decode_bf16_64seq", "bf16", 12, 64, 12, 64, 1280, 1024, graph=True),
        # a few long conversations on a larger model, direct calls
        _decode("decode_bf16_4seq_long", "bf16", 4, 4, 24, 128, 8192, 8000, graph=False),
    ]


def _log_int(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "forward", "decode"])
    if kind == "decode":
        dtype = rng.choice(["f32", "bf16"])
        D = rng.choice([32, 64, 128]) if dtype == "f32" else rng.choice([64, 128])
        H = rng.randint(4, 24)
        B = 1 if dtype == "f32" else _log_int(rng, 1, 128)
        max_len = _log_int(rng, 128, 8192) if dtype == "bf16" else _log_int(rng, 128, 2048)
        layers = rng.choice([2, 4, 12])
        while layers * B * H * max_len * D > 9e8:   # a few GB of caches, as in the listed cases
            max_len = max(128, max_len // 2)
            B = max(1, B // 2)
        return _decode(None, dtype, layers, B, H, D, max_len, rng.randint(max_len // 2, max_len - 1),
                       dtype == "bf16" and rng.random() < 0.5)
    dtype = rng.choice(["f32", "bf16", "bf16", "via_bf16"])
    D = rng.choice([16, 32, 64, 128]) if dtype == "f32" else rng.choice([64, 64, 128])
    rate = 0.1 if dtype != "via_bf16" and rng.random() < 0.3 else 0.0
    layout = "interleaved" if dtype == "bf16" and D == 64 and rate == 0 and rng.random() < 0.3 else "split"
    H = rng.choice([4, 8, 12, 16, 24])
    S = _log_int(rng, 32, 8192 if dtype == "bf16" else 2048)
    B = _log_int(rng, 1, 16)
    # fp32 arithmetic and mask drawing cost more per probability than the tensor cores do
    most = 3e8 if dtype == "f32" or rate else 12e9
    while B * H * S * S > most:
        B, S = max(1, B // 2), (S if B > 1 else S * 2 // 3)
    return _attention(None, kind, dtype, B, H, S, D, rate, layout)


class _State:
    pass


def _prepare_attention(case, seed):
    s = _State()
    B, H, S, D = (case[k] for k in "BHSD")
    s.BH, s.scale, s.rate, s.rng_seed = B * H, D ** -0.5, case["rate"], 42 + seed
    dtype = TORCH_DTYPE[case["dtype"]]
    shape = (B * S, H * D) if case["layout"] == "interleaved" else (s.BH, S, D)
    g = torch.Generator(device="cuda").manual_seed(seed)
    train = case["kind"] == "train"

    def values():
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, 0.5, generator=g)

    s.q, s.k, s.v = values(), values(), values()
    s.out = torch.empty_like(s.q)
    s.lse = torch.empty(s.BH, S, dtype=torch.float32, device="cuda")
    if train:
        s.dout = values()
        s.dq, s.dk, s.dv = (torch.empty_like(s.q) for _ in range(3))
    nbytes = 0
    if case["dtype"] == "via_bf16":
        nbytes = dad.flash_f32_via_bf16_workspace_bytes(s.BH, S, D)
    elif case["dtype"] == "bf16" and train:
        nbytes = dad.flash_backward_bf16_workspace_bytes(s.BH, S, D)
    elif train:
        nbytes = 4 * s.BH * S   # delta
    s.workspace = torch.empty(nbytes // 4, dtype=torch.float32, device="cuda")
    # at head size 64 the bf16 path draws the dropout mask once per step, into this buffer
    s.bits = None
    if s.rate and case["dtype"] == "bf16" and D == 64:
        s.bits = dad.dropout_mask_bits(s.BH, S, s.rate, s.rng_seed)
    return s


def _run_attention(case, s):
    B, H, S, D = (case[k] for k in "BHSD")
    dtype, train = case["dtype"], case["kind"] == "train"
    if dtype == "via_bf16":
        dad.gpu_flash_attention_forward_via_bf16(s.out, s.lse, s.q, s.k, s.v, s.BH, S, D, s.scale, s.workspace)
        if train:
            dad.gpu_flash_attention_backward_via_bf16(s.dq, s.dk, s.dv, s.dout, s.out, s.lse, s.q, s.k, s.v, s.BH,
                                                      S, D, s.scale, s.workspace)
    elif case["layout"] == "interleaved":
        dad.gpu_flash_attention_forward_bf16_interleaved(s.out, s.lse, s.q, s.k, s.v, B, H, S, D, s.scale)
        if train:
            dad.gpu_flash_attention_backward_bf16_interleaved(s.dq, s.dk, s.dv, s.workspace, s.dout, s.out, s.lse,
                                                              s.q, s.k, s.v, B, H, S, D, s.scale)
    else:
        drop = {"rate": s.rate, "seed": s.rng_seed} if s.rate else {}
        forward, backward = dad.gpu_flash_attention_forward, dad.gpu_flash_attention_backward
        if dtype == "bf16":
            forward, backward = dad.gpu_flash_attention_forward_bf16, dad.gpu_flash_attention_backward_bf16
            if s.bits is not None:
                drop["mask_bits"] = dad.dropout_mask_bits(s.BH, S, s.rate, s.rng_seed, out=s.bits)
        forward(s.out, s.lse, s.q, s.k, s.v, s.BH, S, D, s.scale, **drop)
        if train:
            backward(s.dq, s.dk, s.dv, s.workspace, s.dout, s.out, s.lse, s.q, s.k, s.v, s.BH, S, D, s.scale, **drop)
    return (s.out, s.lse, s.dq, s.dk, s.dv) if train else (s.out, s.lse)


def _prepare_decode(case, seed):
    s = _State()
    n, B, H, D, L = case["layers"], case["B"], case["H"], case["D"], case["max_len"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = TORCH_DTYPE[case["dtype"]]
    s.scale = D ** -0.5

    def values(*shape):
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, 1.0, generator=g)

    token = (n, H * D) if case["dtype"] == "f32" else (n, B, H, D)
    s.q, s.k_new, s.v_new = values(*token), values(*token), values(*token)
    s.out = torch.empty_like(s.q)
    if case["dtype"] == "f32":
        s.k, s.v = values(n, H, L, D), values(n, H, L, D)
        s.pos = case["longest"]
        return s
    s.caches = [dad.KVCacheBF16(B, H, L, D) for _ in range(n)]
    for c in s.caches:
        c.k.normal_(0.0, 1.0, generator=g)
        c.v.normal_(0.0, 1.0, generator=g)
    # one length in each of B equal parts of 1..longest, in random order; the layers' lengths lie
    # side by side so that one copy rewinds them all
    part = (torch.rand(B, generator=g, device="cuda") + torch.arange(B, device="cuda"))
    part = part[torch.randperm(B, generator=g, device="cuda")]
    s.start = (1 + part * (case["longest"] / B)).to(torch.int32).clamp_(max=case["longest"]).repeat(n, 1)
    s.lengths = s.start.clone()
    for layer, c in enumerate(s.caches):
        c.lengths = s.lengths[layer]
    s.graph = None
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _token(s, early=True)
            side.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                _token(s, early=True)
        torch.cuda.current_stream().wait_stream(side)
        s.graph = graph
    return s


def _token(s, early):
    """One token for every sequence through all layers, from the state's starting lengths. With
    ``early``, a layer may begin while the layer before it drains (each has its own cache); the
    first layer may not, since the copy ahead of it writes its lengths."""
    s.lengths.copy_(s.start)
    for layer, cache in enumerate(s.caches):
        if early and layer == 1:
            dad.set_decode_early_start(True)
        dad.decode_attention_bf16(s.out[layer], s.q[layer], s.k_new[layer], s.v_new[layer], cache, s.scale)
    if early:
        dad.set_decode_early_start(False)


def _run_decode(case, s):
    if case["dtype"] == "f32":
        for layer in range(case["layers"]):
            dad.decode_attention_f32(s.out[layer], s.q[layer], s.k_new[layer], s.v_new[layer], s.k[layer],
                                     s.v[layer], s.pos, s.scale)
        return s.out, s.k, s.v
    if s.graph is not None:
        s.graph.replay()
    else:
        _token(s, early=False)
    return s.out, s.lengths, [c.k for c in s.caches], [c.v for c in s.caches]


def prepare(case, seed):
    s = _prepare_decode(case, seed) if case["kind"] == "decode" else _prepare_attention(case, seed)
    s.case = case
    return s


def run(state):
    if state.case["kind"] == "decode":
        return _run_decode(state.case, state)
    return _run_attention(state.case, state)


def work(case):
    """Bytes and FLOPs of one pass: every input read once, every output written once; the causal
    half of the products, two in the forward and five in the backward."""
    B, H, D = case["B"], case["H"], case["D"]
    size = TORCH_DTYPE[case["dtype"]].itemsize
    if case["kind"] == "decode":
        if case["dtype"] == "f32":
            rows = case["longest"] + 1
        else:
            rows = B * (1 + (1 + case["longest"]) / 2)   # lengths are spread evenly
        per_layer = rows * 2 * H * D * size + 6 * B * H * D * size
        return {"bytes": case["layers"] * per_layer, "flops": case["layers"] * rows * 4 * H * D}
    S, BH = case["S"], B * H
    pairs = BH * S * (S + 1) / 2
    if case["kind"] == "forward":
        return {"bytes": 4 * BH * S * D * size + 4 * BH * S, "flops": 4 * D * pairs}
    return {"bytes": 8 * BH * S * D * size + 4 * BH * S, "flops": 14 * D * pairs}


def tolerance(case):
    # fp32 sums; elsewhere operands, probabilities and results are rounded to bf16
    return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-2, "max": 0.1}
