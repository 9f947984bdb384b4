"""Soft-capped logits from the head's epilogue against the separate pass, from far above the cap down to nothing."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 300])
@pytest.mark.parametrize("scale", [1e-8, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 0.1, 1.0, 30.0])
def test_every_size_of_logit(M, scale):
    """The epilogue's tangent is within 4e-6 of its value before it is rounded to bf16, the quotient within 2^-22: each rounds another way
    in under one of a hundred places, and one bf16 step there becomes two at most through the product."""
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    K, N, cap = 128, 1040, 15.0
    a, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), (torch.randn(N, K, generator=g, device="cuda") * scale / K**0.5).bfloat16()
    got, want = (torch.empty(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.linear(a, w, got, softcap=cap)
    ops.linear(a, w, want)
    ops.softcap_(want, cap)
    got, want = got.float(), want.float()
    assert (got != want).float().mean().item() <= 1e-2
    assert bool(((got - want).abs() <= 2.0**-6 * want.abs()).all())
