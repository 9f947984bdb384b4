"""Output gate of short or fp32 attention, in the warp-level kernel's epilogue or as a pass behind it, on both sides of each limit of the rule."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,B,H,D,T,gap", [
    (torch.float32, 4, 8, 64, 17, 0), (torch.float32, 4, 8, 64, 17, 3), (torch.float32, 1, 4, 128, 8, 5), (torch.float32, 2, 3, 32, 40, 0),
    (torch.float32, 128, 8, 16, 3, 0), (torch.float32, 129, 8, 16, 3, 0), (torch.float32, 129, 8, 16, 3, 1), (torch.bfloat16, 64, 8, 64, 7, 0),
    (torch.bfloat16, 65, 8, 64, 7, 0), (torch.bfloat16, 65, 8, 64, 8, 0), (torch.bfloat16, 65, 8, 64, 7, 2),
])
def test_gate_equals_the_separate_pass(dt, B, H, D, T, gap):
    """`gap`: rows between the sequences of the output, which a pass over all rows at once could not skip.  fp32: the same arithmetic
    bit for bit; bf16: the sigmoid's last bit before it is rounded, so a bf16 step in one of a thousand places."""
    from diff_gpt_b200 import ops

    C, g = H * D, torch.Generator(device="cuda").manual_seed(B + T + D)
    q = torch.randn((B * T, C), device="cuda", generator=g).to(dt)
    kv = torch.randn((B, 2, H, T, D), device="cuda", generator=g).to(dt)
    gate = torch.randn((B * T, 2 * C), device="cuda", generator=g).to(dt)[:, C:]
    lay = ops.kv_layout(kv[0, 0], kv[0, 1], 2 * H * T * D, T * D, T)
    out = torch.full((2, B, T + gap, C), float("nan"), device="cuda", dtype=dt)
    for y, own in zip(out, (gate, None)):
        ops.fmha_prefill(q, lay, y, B=B, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C, o_batch_stride=(T + gap) * C, o_row_stride=C,
                         kv_len_all=T, causal=True, impl=1, gate=own)
    got, want = out[0, :, :T].reshape(B * T, C), out[1, :, :T].reshape(B * T, C).clone()
    ops.sigmoid_gate(want, gate)
    assert torch.isnan(out[0, :, T:].float()).all()
    if dt == torch.float32:
        assert torch.equal(got, want)
        return
    assert (got != want).float().mean().item() <= 1e-3
    assert bool(((got.float() - want.float()).abs() <= 2.0**-7 * want.float().abs()).all())
