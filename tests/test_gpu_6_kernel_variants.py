"""Sizes at which the kernel variants can go wrong: tile remainders, one to five query tiles (the
barriers and buffers that alternate per tile), every combination of bias form and dropout."""
import pytest
import torch

import oracle
from test_gpu_5_attention_bias_dropout import check, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Sq,Sk,causal", [(64, 130, False), (129, 128, True), (300, 257, False), (400, 400, True),
                                          (640, 131, False)])
@pytest.mark.parametrize("D,code,bias_dtype,p", [
    (64, "matrix", torch.float32, 0.0), (64, "matrix", torch.bfloat16, 0.2), (64, None, None, 0.2),
    (64, "vector", torch.float32, 0.2), (40, "matrix", torch.bfloat16, 0.0), (128, "matrix", torch.float32, 0.2),
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
