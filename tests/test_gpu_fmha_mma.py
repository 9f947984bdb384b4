"""Attention of short sequences with its products in registers (fmha_mma.cu) against float64."""

import pytest
import torch

from diff_gpt_b200 import ops

pytestmark = pytest.mark.gpu

# bf16 in and out: the result's rounding is 1.7e-3 of it, that of the probabilities (whole tiles) and of the gate as much again; 3.1e-3 measured
REL = 4e-3


def _reference(q, k, v, Tq, q_offset, kv_len, causal, gate):
    B, H, _, D = k.shape
    s = q.double().view(B, Tq, H, D).transpose(1, 2) @ k.double().transpose(-1, -2) * D**-0.5
    j = torch.arange(k.shape[2], device="cuda")
    seen = (j[None] < kv_len[:, None])[:, None, None]
    if causal:
        seen = seen & (j[None] <= q_offset + torch.arange(Tq, device="cuda")[:, None])[None, None]
    p = torch.softmax(s.masked_fill(~seen, float("-inf")), -1).nan_to_num(0.0)
    y = (p @ v.double()).transpose(1, 2).reshape(B * Tq, H * D)
    return y if gate is None else y.bfloat16().double() * torch.sigmoid(gate.double())


# (batch, heads, head_dim, keys, query offset): whole tiles and ragged ones around the rule's edges, blocks of 16 rows, few rows
CASES = [(24, 8, 32, 256, 0), (24, 8, 32, 384, 127), (96, 2, 32, 768, 0), (48, 4, 32, 40, 0), (48, 4, 32, 64, 17), (200, 1, 32, 129, 0),
         (64, 3, 32, 700, 650), (1, 3, 32, 33, 0), (2, 8, 32, 128, 0),
         (2, 3, 64, 24, 0), (1, 2, 64, 64, 63), (3, 2, 64, 131, 0), (1, 8, 64, 320, 5), (9, 4, 64, 200, 199)]


@pytest.mark.parametrize("B,H,D,T,off", CASES)
@pytest.mark.parametrize("gated", [False, True])
def test_dense(B, H, D, T, off, gated):
    g = torch.Generator(device="cuda").manual_seed(B + T)
    Tq, C = T - off, H * D
    q, gate = (torch.randn((B * Tq, C), generator=g, device="cuda").bfloat16() for _ in range(2))
    kv = torch.randn((2, B, H, T, D), generator=g, device="cuda").bfloat16()
    kv[:, :, :, ::7] *= 3  # maxima that move late in a row
    y, status = torch.full_like(q, float("nan")), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.fmha_prefill(q, ops.kv_layout(kv[0], kv[1], H * T * D, T * D, T), y, B=B, H=H, Tq=Tq, D=D, q_batch_stride=Tq * C, q_row_stride=C,
                     o_batch_stride=Tq * C, o_row_stride=C, kv_len_all=T, q_offset=off, causal=True, status=status, gate=gate if gated else None)
    ref = _reference(q, kv[0], kv[1], Tq, off, torch.full((B,), T, device="cuda"), True, gate if gated else None)
    assert (y.double() - ref).norm() <= REL * ref.norm() and status.item() == 0


@pytest.mark.parametrize("causal", [True, False])
def test_pages_and_lengths(causal):
    """Scrambled pages, a length per sequence (one of none at all), rows of a wider buffer: on the tcgen05 kernels, by the same reference.  (Lengths of
    dense sequences: test_gpu_prompt_kernels.py.)"""
    g = torch.Generator(device="cuda").manual_seed(3)
    B, H, D, pt, n_pages, Tq = 40, 5, 32, 64, 5, 320
    C = H * D
    pool = torch.randn((B * n_pages + 3, 2, H, pt, D), generator=g, device="cuda").bfloat16()
    table = torch.randperm(B * n_pages + 3, generator=g, device="cuda")[: B * n_pages].to(torch.int32).view(B, n_pages).contiguous()
    kv_len = torch.randint(1, n_pages * pt + 1, (B,), generator=g, device="cuda").to(torch.int32)
    kv_len[0], kv_len[1] = 0, n_pages * pt
    wide = torch.randn((B * Tq, 2 * C), generator=g, device="cuda").bfloat16()
    q, y = wide[:, :C], torch.full((B * Tq, C), float("nan"), device="cuda").bfloat16()
    lay = ops.kv_layout(pool[0, 0], pool[0, 1], 2 * H * pt * D, pt * D, pt, table, pool.shape[0])
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.fmha_prefill(q, lay, y, B=B, H=H, Tq=Tq, D=D, q_batch_stride=Tq * 2 * C, q_row_stride=2 * C, o_batch_stride=Tq * C, o_row_stride=C,
                     kv_len=kv_len, causal=causal, status=status)
    k, v = (pool[table.long(), i].transpose(1, 2).reshape(B, H, n_pages * pt, D) for i in range(2))
    ref = _reference(q, k, v, Tq, 0, kv_len, causal, None)
    assert (y.double() - ref).norm() <= REL * ref.norm() and status.item() == 0
    assert bool((y[:Tq] == 0).all())
