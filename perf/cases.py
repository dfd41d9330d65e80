"""The work that is timed: calls of the public entry points over the range of sizes they serve.

`listed()` names twelve fixed cases, `draw(rng)` gives further ones of the same ranges.  A case is
a dict of plain values; `prepare` makes what a program holds before the call, `run` is one pass,
`work` the bytes and operations a pass cannot do without, `tolerance` what another correct
implementation at the same precision may differ by, `exact` the results in 64 bits.

Kinds of case:
  fwd    attention forward without gradients: inference over a whole sequence (prefill, encoders),
         and with sq = 1 the decoding of one token per sequence against its stored keys and values
  train  attention forward and backward through autograd, as inside a training step
  lion   one optimizer step over a list of parameters
"""
from __future__ import annotations

import math

import torch

from fast_ops_b200.flash_attention import flash_attn_bshd, multi_head_attention
from fast_ops_b200.lion import Lion

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
SIZE = {"f16": 2, "bf16": 2, "f32": 4}
FWD_FLOPS_MOST = 2.0e12    # drawn forward passes stay below half of the largest listed one
TRAIN_FLOPS_MOST = 3.0e11  # the same for forward + backward (3.5 times as many operations)
LION_NUMEL_MOST = 400_000_000


def _attn(kind, name=None, *, b, h, sq, sk, d, dtype="bf16", causal=False, layout="bhsd", kv_heads=0, bias="",
          dropout=0.0):
    case = {"kind": kind, "b": b, "h": h, "sq": sq, "sk": sk, "d": d, "dtype": dtype, "causal": causal,
            "layout": layout, "kv_heads": kv_heads or h, "bias": bias, "dropout": dropout}
    if name:
        case["name"] = name
    return case


def _lion(name=None, *, shapes, param, momentum, tensors=0, smallest=0, largest=0, lr=1e-4, weight_decay=0.1):
    case = {"kind": "lion", "shapes": shapes, "param": param, "momentum": momentum, "tensors": tensors,
            "smallest": smallest, "largest": largest, "lr": lr, "weight_decay": weight_decay}
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest configured attention (B=2, H=4, S=256, head_dim 64): the call itself counts.
        _attn("fwd", "fwd_small_f16", b=2, h=4, sq=256, sk=256, d=64, dtype="f16"),
        # One layer of a small language model's training step: the configured GPT-2-small shape.
        _attn("train", "train_s1024_d64", b=8, h=12, sq=1024, sk=1024, d=64, causal=True),
        # The reference's own benchmark shape (1, 12, S, 128) without a mask: an encoder, one sequence.
        _attn("fwd", "fwd_s4096_full", b=1, h=12, sq=4096, sk=4096, d=128),
        # Prefill of a long context: the configured long-context shape, the largest attention here.
        _attn("fwd", "fwd_s16384_causal", b=2, h=32, sq=16384, sk=16384, d=128, causal=True),
        # One layer of a 7B-sized model's training step at a 4k context.
        _attn("train", "train_s4096_d128", b=2, h=32, sq=4096, sk=4096, d=128, causal=True),
        # Cross attention of an encoder-decoder or image model: ragged lengths, a head_dim between
        # the kernels' own, fp16, (B, S, H, D) tensors.
        _attn("train", "train_cross_ragged_d80", b=4, h=12, sq=1000, sk=1531, d=80, dtype="f16", layout="bshd"),
        # Training with linear position biases, the reference's tested length 3072.
        _attn("train", "train_alibi_s3072", b=2, h=16, sq=3072, sk=3072, d=128, causal=True, layout="bshd",
              bias="1h1k"),
        # Training with a learned relative-position bias matrix and attention dropout.
        _attn("train", "train_bias_dropout_d64", b=2, h=16, sq=2048, sk=2048, d=64, layout="bshd", bias="1hqk",
              dropout=0.1),
        # Decoding: one token for each of four sequences with 4096 tokens of context.
        _attn("fwd", "decode_b4_k4096", b=4, h=32, sq=1, sk=4096, d=128),
        # The optimizer step of a GPT-2-medium-shaped list: fp32 weights, bf16 momentum.
        _lion("lion_gpt2_medium", shapes="gpt2_medium", param="f32", momentum="bf16"),
        # The reference's smallest optimizer benchmark point: the launch itself counts.
        _lion("lion_8192_bf16", shapes="spread", param="bf16", momentum="bf16", tensors=1, smallest=8192,
              largest=8192),
        # Four layers of the configured Llama-7B list, all bf16.
        _lion("lion_llama7b_4_layers", shapes="llama7b_layers", param="bf16", momentum="bf16", lr=3e-5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length: half of them multiples of 64, half any number."""
    n = _log_int(rng, lo, hi)
    return max(64, n // 64 * 64) if rng.random() < 0.5 else n


def draw(rng):
    pick = rng.random()
    if pick < 0.25:
        numel = [8, 1_000_000, 16_000_000]
        while True:
            tensors = _log_int(rng, 1, 300)
            smallest = _log_int(rng, numel[0], numel[1])
            largest = max(smallest, _log_int(rng, 1024, numel[2]))
            param, momentum = rng.choice([("f32", "bf16"), ("f32", "f32"), ("bf16", "bf16"), ("f16", "f16")])
            case = _lion(shapes="spread", param=param, momentum=momentum, tensors=tensors, smallest=smallest,
                         largest=largest, lr=rng.choice([1e-4, 3e-5]), weight_decay=rng.choice([0.0, 0.1]))
            if sum(math.prod(s) for s in _lion_shapes(case)) <= LION_NUMEL_MOST:
                return case
    d = rng.choice([64, 64, 128, 128, 128, 32, 40, 80, 96])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    layout = rng.choice(["bhsd", "bshd"])
    if pick < 0.40:
        h = rng.choice([8, 12, 16, 32, 40])
        b = _log_int(rng, 1, 32)
        sk = _length(rng, 128, max(129, min(32768, 4_000_000 // (b * h))))
        return _attn("fwd", b=b, h=h, sq=1, sk=sk, d=d, dtype=dtype, layout=layout, kv_heads=rng.choice([h, h, 1]))
    most = FWD_FLOPS_MOST if pick < 0.65 else TRAIN_FLOPS_MOST
    while True:
        b, h = _log_int(rng, 1, 32), rng.choice([4, 8, 12, 16, 32])
        sq = _length(rng, 64, 16384)
        causal = rng.random() < 0.6
        sk = sq if causal or rng.random() < 0.6 else _length(rng, 64, 8192)
        kv_heads = rng.choice([h, h, h, 1])
        bias, dropout = "", 0.0
        if rng.random() < 0.3:
            bias = rng.choice(["1h1k", "b11k", "1hqk"])
        if pick >= 0.65 and rng.random() < 0.3:
            dropout = 0.1
        if bias == "1hqk" and h * sq * sk > 1 << 28:
            continue
        case = _attn("fwd" if pick < 0.65 else "train", b=b, h=h, sq=sq, sk=sk, d=d, dtype=dtype, causal=causal,
                     layout=layout, kv_heads=kv_heads, bias=bias, dropout=dropout)
        if _fwd_flops(case) <= most and b * h * max(sq, sk) * d <= 1 << 28:
            return case


# ---- parameter lists -----------------------------------------------------------------------------

def _lion_shapes(case):
    if case["shapes"] == "gpt2_medium":
        c = 1024
        block = [(c, 3 * c), (3 * c,), (c, c), (c,), (c, 4 * c), (4 * c,), (4 * c, c), (c,), (c,), (c,), (c,), (c,)]
        return [(50257, c), (1024, c)] + block * 24 + [(c,), (c,)]
    if case["shapes"] == "llama7b_layers":
        c, f = 4096, 11008
        return [(c, c), (c, c), (c, c), (c, c), (f, c), (f, c), (c, f), (c,), (c,)] * 4
    n, lo, hi = case["tensors"], case["smallest"], case["largest"]
    shapes = []
    for i in range(n):  # spread over the logarithm, in no sorted order
        t = ((i * 0.6180339887498949) % 1.0) if n > 1 else 0.0
        shapes.append((int(round(lo * (hi / lo) ** t)),))
    return shapes


def _prepare_lion(case, seed):
    """Parameters, gradients and momentum as views of one buffer each (flat parameter storage,
    gradient buckets), every tensor on a 512-byte boundary as the caching allocator places them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pdt, mdt = DTYPES[case["param"]], DTYPES[case["momentum"]]
    shapes = _lion_shapes(case)
    offsets, at = [], 0
    for s in shapes:
        offsets.append(at)
        at += (math.prod(s) + 255) // 256 * 256
    flat_p = torch.empty(at, dtype=pdt, device="cuda").normal_(0.0, 0.02, generator=gen)
    flat_g = torch.empty(at, dtype=pdt, device="cuda").normal_(0.0, 1e-3, generator=gen)
    flat_m = torch.empty(at, dtype=mdt, device="cuda").normal_(0.0, 5e-4, generator=gen)
    params = []
    for s, o in zip(shapes, offsets):
        n = math.prod(s)
        p = torch.nn.Parameter(flat_p[o:o + n].view(s))
        p.grad = flat_g[o:o + n].view(s)
        params.append(p)
    opt = Lion(params, lr=case["lr"], betas=(0.9, 0.99), weight_decay=case["weight_decay"], momentum_dtype=mdt)
    for p, o in zip(params, offsets):
        opt.state[p]["exp_avg"] = flat_m[o:o + p.numel()].view(p.shape)
    return {"kind": "lion", "opt": opt, "params": flat_p, "momentum": flat_m}


# ---- attention -----------------------------------------------------------------------------------

def _prepare_attn(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    b, h, sq, sk, d = (case[k] for k in ("b", "h", "sq", "sk", "d"))
    train = case["kind"] == "train"
    bshd = case["layout"] == "bshd"

    def tensor(heads, s):
        shape = (b, s, heads, d) if bshd else (b, heads, s, d)
        return torch.empty(shape, dtype=dt, device="cuda").normal_(generator=gen)

    q, k, v = tensor(h, sq), tensor(case["kv_heads"], sk), tensor(case["kv_heads"], sk)
    state = {"kind": case["kind"], "bshd": bshd, "h": h, "q": q, "k": k, "v": v, "causal": case["causal"],
             "dropout": case["dropout"], "bias": None}
    if train:
        for t in (q, k, v):
            t.requires_grad_()
        state["grad_out"] = tensor(h, sq)
    if case["bias"] == "1h1k":  # linear position bias: a slope per head times the key's position
        slopes = torch.exp2(-8.0 * torch.arange(1, h + 1, device="cuda", dtype=torch.float32) / h)
        state["bias"] = (slopes[:, None] * torch.arange(1 - sk, 1, device="cuda", dtype=torch.float32)).view(1, h, 1, sk)
    elif case["bias"] == "b11k":  # key padding: the last few keys of each sequence are masked
        keys = torch.arange(sk, device="cuda")
        lens = sk - torch.randint(0, max(1, sk // 4), (b, 1), generator=gen, device="cuda")
        state["bias"] = torch.zeros(b, sk, device="cuda").masked_fill(keys >= lens, float("-inf")).view(b, 1, 1, sk)
    elif case["bias"] == "1hqk":  # relative-position bias, in the input type as a model keeps it
        state["bias"] = torch.empty(1, h, sq, sk, dtype=dt, device="cuda").normal_(generator=gen)
    if case["dropout"] > 0:
        torch.cuda.manual_seed(seed)  # the mask comes from the device's generator
    return state


def _attention(state):
    q, k, v, h = state["q"], state["k"], state["v"], state["h"]
    if state["bshd"]:
        if k.shape[2] != h:
            k, v = (t.expand(-1, -1, h, -1) for t in (k, v))
        return flash_attn_bshd(q, k, v, state["bias"], state["causal"], state["dropout"])
    if k.shape[1] != h:
        k, v = (t.expand(-1, h, -1, -1) for t in (k, v))
    return multi_head_attention(q, k, v, causal=state["causal"], bias=state["bias"], dropout_p=state["dropout"])


def prepare(case, seed):
    return _prepare_lion(case, seed) if case["kind"] == "lion" else _prepare_attn(case, seed)


def run(state):
    if state["kind"] == "lion":
        state["opt"].step()
        return state["params"], state["momentum"]
    if state["kind"] == "fwd":
        with torch.no_grad():
            return _attention(state)
    o = _attention(state)
    dq, dk, dv = torch.autograd.grad(o, (state["q"], state["k"], state["v"]), state["grad_out"])
    return o, dq, dk, dv


def _exact_lion(case, seed):
    state = _prepare_lion(case, seed)
    opt = state["opt"]
    lr, wd, (b1, b2) = case["lr"], case["weight_decay"], (0.9, 0.99)
    p_out, m_out = state["params"].double(), state["momentum"].double()
    at = 0
    for p in opt.param_groups[0]["params"]:
        n = p.numel()
        g = p.grad.reshape(-1).double()
        pn, mn = p_out[at:at + n], m_out[at:at + n]
        pn.mul_(1 - lr * wd).sub_((mn * b1 + g * (1 - b1)).sign_(), alpha=lr)
        mn.mul_(b2).add_(g, alpha=1 - b2)
        at += (n + 255) // 256 * 256
    return p_out, m_out


def _exact_head(q, k, v, bias, causal, grad_out):
    """One head in 64 bits, a slab of query rows at a time: (o,) or (o, dq, dk, dv)."""
    sq, d = q.shape
    sk = k.shape[0]
    q, k, v = q.double(), k.double(), v.double()
    o = torch.empty_like(q)
    dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    scale = 1.0 / math.sqrt(d)
    rows = max(64, (1 << 26) // sk)
    for r in range(0, sq, rows):
        e = min(sq, r + rows)
        keys = min(sk, e) if causal else sk
        s = (q[r:e] @ k[:keys].T) * scale
        if bias is not None:
            s += (bias[r:e, :keys] if bias.shape[0] > 1 else bias[:, :keys]).double()
        if causal:
            above = torch.arange(keys, device=q.device)[None, :] > torch.arange(r, e, device=q.device)[:, None]
            s.masked_fill_(above, float("-inf"))
        p = torch.softmax(s, dim=-1)
        o[r:e] = p @ v[:keys]
        if grad_out is not None:
            g = grad_out[r:e].double()
            ds = p * (g @ v[:keys].T - (g * o[r:e]).sum(-1, keepdim=True))
            dq[r:e] = (ds @ k[:keys]) * scale
            dk[:keys] += (ds.T @ q[r:e]) * scale
            dv[:keys] += p.T @ g
    return (o,) if grad_out is None else (o, dq, dk, dv)


def exact(case, seed):
    """The outputs of the first pass in 64 bits.  None with dropout (the mask is the framework's own)."""
    if case["kind"] == "lion":
        return _exact_lion(case, seed)
    if case["dropout"] > 0:
        return None
    state = _prepare_attn(case, seed)
    bshd, h, bias = state["bshd"], case["h"], state["bias"]

    def heads(t):
        return t.detach().transpose(1, 2) if bshd else t.detach()

    q, k, v = heads(state["q"]), heads(state["k"]), heads(state["v"])
    grad_out = heads(state["grad_out"]) if "grad_out" in state else None
    outs = [torch.zeros(t.shape, dtype=torch.float64, device=t.device)
            for t in ((q,) if grad_out is None else (q, q, k, v))]
    for b in range(case["b"]):
        for i in range(h):
            j = i % k.shape[1]
            one = None if bias is None else bias[b % bias.shape[0], i % bias.shape[1]]
            got = _exact_head(q[b, i], k[b, j], v[b, j], one, case["causal"],
                              None if grad_out is None else grad_out[b, i])
            for out, x, at in zip(outs, got, (i, i, j, j)):
                out[b, at] += x  # a shared key/value head collects its gradient from every query head
    if bshd:
        outs = [t.transpose(1, 2).contiguous() for t in outs]
    return outs[0] if grad_out is None else tuple(outs)


def _fwd_flops(case):
    """Two matmuls over the (query, key) pairs that the mask leaves (causal: key <= query)."""
    sq, sk = case["sq"], case["sk"]
    pairs = sq * sk
    if case["causal"]:
        full = min(sq, sk)
        pairs = full * (full + 1) // 2 + max(0, sq - sk) * sk
    return 4.0 * case["b"] * case["h"] * pairs * case["d"]


def work(case):
    if case["kind"] == "lion":
        n = sum(math.prod(s) for s in _lion_shapes(case))
        # p, g, m read; p, m written; about ten operations per element
        return {"bytes": n * (3 * SIZE[case["param"]] + 2 * SIZE[case["momentum"]]), "flops": 10.0 * n}
    e = SIZE[case["dtype"]]
    b, h, sq, sk, d = (case[k] for k in ("b", "h", "sq", "sk", "d"))
    q, kv = b * h * sq * d * e, 2 * b * case["kv_heads"] * sk * d * e
    bias = {"": 0, "1h1k": 4 * h * sk, "b11k": 4 * b * sk, "1hqk": e * h * sq * sk}[case["bias"]]
    moved = q + kv + bias + q  # Q, K, V, bias in; O out
    flops = _fwd_flops(case)
    if case["kind"] == "train":
        moved += q + q + kv  # dO in; dQ, dK, dV out
        flops *= 3.5         # the backward's five matmuls against the forward's two
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["kind"] == "lion":
        return "exact"  # the update is defined rounding by rounding
    # against the same path in 64 bits every output is off by 2.1e-3 to 2.5e-3 in bf16 and 2.6e-4 to
    # 3.1e-4 in fp16 (probabilities and results rounded to the input type): four times that
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1.25e-3}
