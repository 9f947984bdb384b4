"""Attention of bf16 queries over dense keys of any length with an fp32 output: fp32 probabilities, whatever the number of keys."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("T", [20, 24, 32, 33, 200, 777, 1100])
def test_error_is_that_of_fp32_sums(T, D):
    """exp2 within 2 ulp, sums of T terms in fp32 tiles of 32: 2^-19 of sum p |v|.  (Probabilities as a pair of bf16 numbers: 2^-17 and more.)"""
    from diff_gpt_b200 import ops

    B, H = 2, 3
    C, g = H * D, torch.Generator(device="cuda").manual_seed(T + D)
    q = torch.randn((B, T, H, D), device="cuda", generator=g).bfloat16()
    kv = torch.randn((B, 2, H, T, D), device="cuda", generator=g).bfloat16()
    y = torch.full((B, T, H, D), float("nan"), device="cuda")
    lse = torch.empty((B, T, H), device="cuda")
    ops.fmha_prefill(q, ops.kv_layout(kv[0, 0], kv[0, 1], 2 * H * T * D, T * D, T), y, B=B, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C,
                     o_batch_stride=T * C, o_row_stride=C, kv_len_all=T, causal=True, lse=lse)
    s = torch.einsum("bihd,bhjd->bhij", q.double(), kv[:, 0].double()) * D**-0.5
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    p, v = torch.softmax(s, -1), kv[:, 1].double()
    want, terms = (torch.einsum("bhij,bhjd->bihd", p, x) for x in (v, v.abs()))
    assert bool(((y.double() - want).abs() <= 2.0**-19 * terms).all()), ((y.double() - want).abs() / terms).max().item()
    assert (lse.double() - torch.logsumexp(s, -1).transpose(1, 2)).abs().max().item() <= 1e-5
