"""Attention over dense keys of any length on the tensor-core kernels, the output gate in the attention epilogue, and the
soft-cap in the head GEMM's: each against the separate passes or float64."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, H, T, D, cap, dt, seed=0):
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(seed + T + D)
    C = H * D
    q = torch.randn((B * T, C), device="cuda", generator=g).to(dt)
    kv = torch.randn((B, 2, H, cap, D), device="cuda", generator=g).to(dt)
    kv[:, :, :, T:] = float("nan")  # cache slots behind the keys may hold anything
    gate = torch.randn((B * T, 2 * C), device="cuda", generator=g).to(dt)[:, C:]  # a slice of a wider projection
    lay = ops.kv_layout(kv[0, 0], kv[0, 1], 2 * H * cap * D, cap * D, cap)
    return q, kv, gate, lay


def _attend(q, lay, B, H, T, D, gate=None, impl=0):
    from diff_gpt_b200 import ops

    y = torch.full_like(q, float("nan"))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    C = H * D
    ops.fmha_prefill(q, lay, y, B=B, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C, o_batch_stride=T * C, o_row_stride=C,
                     kv_len_all=T, causal=True, impl=impl, status=status, gate=gate)
    assert status.item() == 0
    return y


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("T,cap", [(1, 1), (17, 17), (127, 127), (129, 129), (200, 203), (1023, 1023), (1025, 1040), (1400, 1400)])
def test_dense_keys_of_any_length(T, cap, D):
    B, H = 2, 3
    q, kv, _, lay = _inputs(B, H, T, D, cap, torch.bfloat16)
    got = _attend(q, lay, B, H, T, D).view(B, T, H, D).transpose(1, 2).double()
    k, v = kv[:, 0, :, :T].double(), kv[:, 1, :, :T].double()
    s = q.view(B, T, H, D).transpose(1, 2).double() @ k.transpose(-1, -2) / math.sqrt(D)
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    p = torch.softmax(s, -1)
    want = p @ v
    # output rounded to bf16 (2^-9 of the value) and probabilities rounded to bf16 before the product (2^-9 of sum p |v|)
    bound = 2.0**-8 * want.abs() + 2.0**-8 * (p @ v.abs()) + 1e-6
    assert bool(((got - want).abs() <= bound).all())


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("T", [33, 127, 300, 777, 1400])
def test_probabilities_of_dense_keys_keep_more_than_bf16(T, D):
    """Against the warp-level kernel (probabilities in fp32): sums that agree to 2^-16 or so round to different bf16 numbers in
    under one of a hundred places, a step of 2^-8 each: 5e-4 in the norm.  Probabilities rounded to bf16 give 1.4e-3."""
    B, H = 2, 3
    q, _, _, lay = _inputs(B, H, T, D, T, torch.bfloat16)
    a, b = (_attend(q, lay, B, H, T, D, impl=impl).float() for impl in (0, 1))
    assert ((a - b).norm() / b.norm()).item() <= 5e-4


@pytest.mark.parametrize("dt,D,T,cap,impl", [
    (torch.bfloat16, 32, 130, 256, 2), (torch.bfloat16, 32, 130, 256, 3), (torch.bfloat16, 64, 77, 77, 0), (torch.bfloat16, 128, 300, 384, 2),
    (torch.bfloat16, 128, 300, 384, 3), (torch.bfloat16, 64, 1100, 1100, 0), (torch.bfloat16, 16, 40, 40, 0), (torch.float32, 16, 90, 90, 0),
    (torch.float32, 128, 33, 64, 0),
])
def test_gate_in_the_epilogue_equals_the_separate_pass(dt, D, T, cap, impl):
    from diff_gpt_b200 import ops

    B, H = 2, 2
    q, _, gate, lay = _inputs(B, H, T, D, cap, dt)
    want = _attend(q, lay, B, H, T, D, impl=impl)
    ops.sigmoid_gate(want, gate)
    got = _attend(q, lay, B, H, T, D, gate=gate, impl=impl)
    if dt == torch.float32:
        assert torch.equal(got, want)
    # bf16: the sigmoid to 2 ulp of fp32 instead of 1, the same bf16 value but for a neighbour on a rounding boundary
    assert (got != want).float().mean().item() <= 1e-3
    assert bool(((got.float() - want.float()).abs() <= 2.0**-7 * want.float().abs()).all())


@pytest.mark.parametrize("M,N,K", [(1, 16, 8), (130, 272, 72), (300, 512, 256)])
def test_softcap_in_the_head_gemm(M, N, K):
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn((N, K), device="cuda", generator=g).to(torch.bfloat16)
    want, got = (torch.empty((M, N), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.linear(a, w, want)
    ops.softcap_(want, 15.0)
    ops.linear(a, w, got, softcap=15.0)
    # tanh to 2e-7 instead of 1e-7: the same bf16 value but for a neighbour where it lies on a rounding boundary
    differ = got != want
    assert differ.float().mean().item() <= 1e-3
    assert bool(((got.float() - want.float()).abs() <= 2.0**-7 * want.float().abs()).all())
