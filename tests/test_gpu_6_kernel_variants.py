"""Sizes at which the kernel variants can go wrong: tile remainders, one to five query tiles (the
barriers and buffers that alternate per tile), every compiled combination of bias form and dropout."""
import pytest
import torch

import oracle
from fast_ops_b200.flash_attention import flash_attention_forward
from test_gpu_5_attention_bias_dropout import check, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Sq,Sk,causal", [(64, 130, False), (129, 128, True), (300, 257, False), (400, 400, True),
                                          (640, 131, False)])
@pytest.mark.parametrize("D,code,bias_dtype,p", [
    (64, "matrix", torch.float32, 0.0), (64, "matrix", torch.bfloat16, 0.2), (64, None, None, 0.2),
    (64, "vector", torch.float32, 0.2), (40, "matrix", torch.bfloat16, 0.0), (128, "matrix", torch.float32, 0.2),
    (64, "vector", torch.float32, 0.0), (64, None, None, 0.0), (128, "vector", torch.bfloat16, 0.0),
    (128, "vector", torch.float32, 0.2), (128, "matrix", torch.bfloat16, 0.0), (128, None, None, 0.2),
    (96, None, None, 0.0), (96, "vector", torch.float32, 0.0), (128, None, None, 0.0),
])
def test_backward_bias_and_dropout_variants(cuda_device, Sq, Sk, causal, D, code, bias_dtype, p):
    B, H = 2, 2
    gen = torch.Generator().manual_seed(Sq * 1000 + Sk + D)
    q, dout = (torch.randn(B, H, Sq, D, generator=gen).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, H, Sk, D, generator=gen).bfloat16() for _ in range(2))
    bias = None
    if code is not None:
        bias = torch.randn(1, H, Sq if code == "matrix" else 1, Sk, generator=gen).to(bias_dtype).float()
        if code == "matrix":
            bias[0, 0, Sq // 2, ::3] = float("-inf")  # masked entries in one row
    # next to a boundary between a kept and a dropped run of the hash: a mixed mask
    rng = (0, 16773120 + 4096 - (B * H * Sq * Sk) // 2 // 4 * 4) if p > 0 else None
    got, _, same, _ = run_case(cuda_device, q, k, v, dout, causal, bias, p, rng, bias_dtype or torch.float32)
    keep = oracle.dropout_mask(p, B, H, Sq, Sk, *rng) if p > 0 else None
    out, _, dq, dk, dv = oracle.attention_ex(q, k, v, bias=bias, keep_mask=keep, dropout_p=p, causal=causal, dout=dout)
    check(got, same, (out, dq, dk, dv), f"D={D} {code} p={p}")


@pytest.mark.parametrize("B,H,Sk,D,dtype,kv_heads,layout", [
    (1, 1, 1, 64, torch.bfloat16, 1, "bhsd"), (2, 3, 7, 128, torch.float16, 3, "bhsd"),
    (1, 2, 255, 40, torch.bfloat16, 2, "bshd"), (3, 5, 511, 128, torch.bfloat16, 1, "bhsd"),
    (1, 4, 513, 64, torch.float16, 1, "bshd"), (2, 2, 1024, 8, torch.float16, 2, "bhsd"),
    (1, 8, 4099, 128, torch.bfloat16, 8, "bshd"), (1, 6, 3000, 96, torch.float16, 1, "bhsd"),
    (2, 3, 2049, 80, torch.bfloat16, 3, "bhsd"), (40, 8, 600, 64, torch.bfloat16, 8, "bhsd"),
])
def test_one_query_row(cuda_device, B, H, Sk, D, dtype, kv_heads, layout):
    """Decoding: keys split over warps and cluster CTAs, ragged ends, shared K/V heads, LSE."""
    gen = torch.Generator(device=cuda_device).manual_seed(Sk + D)

    def make(heads, s):
        shape = (B, s, heads, D) if layout == "bshd" else (B, heads, s, D)
        t = torch.empty(shape, device=cuda_device).normal_(generator=gen).to(dtype)
        return t.transpose(1, 2) if layout == "bshd" else t

    q, k, v = make(H, 1), make(kv_heads, Sk), make(kv_heads, Sk)
    k[:, :, Sk // 2] *= 4  # a maximum in the middle of a split
    k, v = k.expand(-1, H, -1, -1), v.expand(-1, H, -1, -1)
    o, lse = flash_attention_forward(q, k, v, return_lse=True)
    s = (q.double() @ k.double().transpose(-1, -2)) / D ** 0.5
    want = torch.softmax(s, -1) @ v.double()
    # fp32 throughout, one rounding of the result (half an ulp of 8 significant bits in bf16, 11 in
    # fp16: 2^-8 and 2^-11 of the value); sums of Sk terms of size <= 5 in fp32 stay within 1e-5
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert ((o.double() - want).abs() <= 1.01 * rel * want.abs() + 2e-5).all()
    assert torch.allclose(lse.double(), torch.logsumexp(s, -1), atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("B,H,shared", [(1, 8, False), (1, 8, True), (4, 32, False), (4, 32, True), (32, 12, False),
                                        (32, 12, True), (16, 40, False), (16, 40, True), (64, 33, True)])
@pytest.mark.parametrize("Sk", [1, 17, 64, 129, 300, 513, 1000, 1024, 1025])
@pytest.mark.parametrize("D", [40, 128])
def test_one_query_row_shapes(cuda_device, B, H, shared, Sk, D):
    """Few to many heads, few to many keys: one or four heads per CTA, two to eight warps, one to eight
    CTAs per head.  Every shape against the same call in 64 bits."""
    gen = torch.Generator(device=cuda_device).manual_seed(B + Sk)
    q = torch.empty(B, H, 1, D, device=cuda_device).normal_(generator=gen).bfloat16()
    k, v = (torch.empty(B, 1 if shared else H, Sk, D, device=cuda_device).normal_(generator=gen).bfloat16()
            .expand(B, H, Sk, D) for _ in range(2))
    o, lse = flash_attention_forward(q, k, v, return_lse=True)
    for b in range(0, B, 5):  # a slice at a time: the 64-bit copies stay small
        s = (q[b].double() @ k[b].double().transpose(-1, -2)) / D ** 0.5
        want = torch.softmax(s, -1) @ v[b].double()
        # one rounding to 8 significant bits; fp32 sums of Sk terms stay within 2e-5
        assert ((o[b].double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 2e-5).all()
        assert torch.allclose(lse[b].double(), torch.logsumexp(s, -1), atol=1e-4, rtol=1e-5)


def test_one_query_row_causal_sees_key_zero_and_graph_replay(cuda_device):
    q, k, v = (torch.randn(2, 3, s, 64, device=cuda_device, dtype=torch.bfloat16) for s in (1, 700, 700))
    assert torch.equal(flash_attention_forward(q, k, v, causal=True), v[:, :, :1])
    eager = flash_attention_forward(q, k, v)
    out = torch.empty_like(q)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        flash_attention_forward(q, k, v, out=out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


@pytest.mark.parametrize("bad", ["batch_stride_0", "row_stride", "base"])
def test_one_query_row_refuses_what_the_tiled_path_refuses(cuda_device, bad):
    q = torch.randn(2, 3, 1, 64, device=cuda_device, dtype=torch.bfloat16)
    k = torch.randn(2, 3, 64, 64, device=cuda_device, dtype=torch.bfloat16)
    if bad == "batch_stride_0":
        k = k[:1].expand(2, -1, -1, -1)
    elif bad == "row_stride":
        k = torch.randn(2, 3, 64, 68, device=cuda_device, dtype=torch.bfloat16)[..., :64]
    else:
        k = torch.randn(2 * 3 * 64 * 64 + 4, device=cuda_device, dtype=torch.bfloat16)[4:].view(2, 3, 64, 64)
    with pytest.raises(RuntimeError):
        flash_attention_forward(q, k, k)


def test_a_thread_without_a_cuda_context_can_call(cuda_device):
    """The tensor maps are encoded by a driver call that needs a context on the calling thread."""
    import threading

    q = torch.randn(1, 2, 136, 64, device=cuda_device, dtype=torch.bfloat16)
    out, result = torch.empty_like(q), []
    want = flash_attention_forward(q, q, q)
    torch.cuda.synchronize()

    def call():
        try:
            result.append(flash_attention_forward(q, q, q, out=out, softmax_scale=0.125))
        except RuntimeError as e:
            result.append(e)

    t = threading.Thread(target=call)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert result[0] is out and torch.equal(out, want)


@pytest.mark.parametrize("D", [72, 80, 96, 104])
@pytest.mark.parametrize("impl", ["ws64", "ws64s"])
def test_head_dims_around_the_96_column_kernels(cuda_device, D, impl):
    """72 to 96 run matmuls of width 96, 104 those of width 128: forward and backward against the oracle."""
    import fast_ops_b200._lib as L

    B, H, Sq, Sk = 1, 2, 260, 330
    gen = torch.Generator().manual_seed(D)
    q, dout = (torch.randn(B, H, Sq, D, generator=gen).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, H, Sk, D, generator=gen).bfloat16() for _ in range(2))
    L.attn_configure(impl=impl)
    try:
        got, _, same, _ = run_case(cuda_device, q, k, v, dout, False, None, 0.0, None)
    finally:
        L.attn_configure(impl="auto")
    out, _, dq, dk, dv = oracle.attention_ex(q, k, v, causal=False, dout=dout)
    check(got, same, (out, dq, dk, dv), f"D={D} {impl}")
