"""The order in which the bias kernel takes the keys: biases that move the row maximum at every step of
one order or the other, runs of masked keys that are the first thing a row sees, an odd number of
64-key steps, query tiles with different numbers of steps."""
import pytest
import torch

import fast_ops_b200._lib as L
import oracle
from fast_ops_b200.flash_attention import flash_attention_forward
from helpers import attention_dout, attention_inputs
from test_gpu_5_attention_bias_dropout import check, run_case

pytestmark = pytest.mark.gpu

SHAPES = [(384, 384, True), (640, 640, True), (512, 512, False), (700, 577, True), (300, 540, False),
          (600, 450, True), (200, 64, False), (130, 192, True)]


def make_bias(kind, B, H, Sq, Sk):
    i, j = torch.arange(Sq)[:, None].float(), torch.arange(Sk).float()
    slope = torch.tensor([0.5, 0.05])[:, None, None]  # per head: the maximum moves by 32 and 3.2 a step
    if kind == "rising":
        return (slope * (j - Sk + 1)).view(1, H, 1, Sk)
    if kind == "falling":
        return (-slope * j).view(1, H, 1, Sk)
    if kind == "peak":
        return (-slope * (j - Sk // 2).abs()).view(1, H, 1, Sk)
    if kind.startswith("padded"):  # per sequence: the last keys masked, by -inf or by a large number
        bias = torch.zeros(B, 1, 1, Sk)
        masked = -1e9 if kind.endswith("finite") else float("-inf")
        for b, n in enumerate([1, 64] if kind.startswith("padded_short") else [130, min(300, Sk - 8)]):
            bias[b, ..., Sk - min(n, Sk - 8):] = masked
        return bias
    if kind == "left_padded":
        bias = torch.zeros(B, 1, 1, Sk)
        for b, n in enumerate([70, 200]):
            bias[b, ..., :min(n, Sk - 8)] = float("-inf")
        return bias
    if kind == "distance":  # largest on the diagonal
        return (-slope * (i - j).abs()).view(1, H, Sq, Sk)
    assert kind == "falling_matrix"
    return (-slope * (j + 0 * i)).view(1, H, Sq, Sk)


@pytest.mark.parametrize("Sq,Sk,causal", SHAPES, ids=lambda x: str(x))
@pytest.mark.parametrize("kind", ["rising", "falling", "peak", "padded_short", "padded_long", "padded_long_finite",
                                  "left_padded", "distance", "falling_matrix"])
@pytest.mark.parametrize("D,dtype,bias_dtype,p", [(64, torch.float16, torch.float16, 0.0),
                                                  (128, torch.bfloat16, torch.float32, 0.2)], ids=["d64", "d128"])
def test_bias_that_moves_the_maximum(cuda_device, Sq, Sk, causal, kind, D, dtype, bias_dtype, p):
    if causal and kind == "left_padded":
        pytest.skip("rows without a visible key: test_fully_masked_rows_give_zero")
    B = H = 2
    q, k, v = attention_inputs(Sq + Sk + D, B, H, Sq, Sk, D, dtype)
    dout = attention_dout(Sq + D, B, H, Sq, D, dtype)
    if kind.endswith("finite"):
        bias_dtype = torch.float32
    bias = make_bias(kind, B, H, Sq, Sk).to(bias_dtype).float()
    rng = (0, 16773120 + 4096 - (B * H * Sq * Sk) // 2 // 4 * 4) if p > 0 else None
    L.attn_configure(impl="ws64")
    try:
        got, lse, same, _ = run_case(cuda_device, q, k, v, dout, causal, bias, p, rng, bias_dtype)
    finally:
        L.attn_configure(impl="auto")
    keep = oracle.dropout_mask(p, B, H, Sq, Sk, *rng) if p > 0 else None
    out, lse_o, dq, dk, dv = oracle.attention_ex(q, k, v, bias=bias, keep_mask=keep, dropout_p=p, causal=causal, dout=dout)
    check(got, same, (out, dq, dk, dv), f"{kind} {Sq}x{Sk}")
    assert torch.allclose(lse.cpu(), lse_o, atol=2e-3, rtol=1e-3)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("form", ["vector", "matrix"])
def test_rows_masked_by_a_large_finite_bias(cuda_device, dtype, form):
    """Every key of a row at -1e9: in fp32 the scores vanish beside it, so the row is the mean of V."""
    B, H, Sq, Sk, D = 1, 2, 300, 450, 64
    q, k, v = (t.to(cuda_device) for t in attention_inputs(5, B, H, Sq, Sk, D, dtype))
    bias = torch.full((1, 1, 1 if form == "vector" else Sq, Sk), -1e9, device=cuda_device)
    L.attn_configure(impl="ws64")
    try:
        o = flash_attention_forward(q, k, v, bias=bias)
    finally:
        L.attn_configure(impl="auto")
    want = v.double().mean(2, keepdim=True).expand_as(o)
    # the weights are exactly 1: fp32 sums of Sk terms below 5, one rounding of the result
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert ((o.double() - want).abs() <= eps * want.abs() + 1e-5).all()
