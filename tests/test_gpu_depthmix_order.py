"""Every form of the depth-mix kernel adds in one order: a row's result does not depend on how many rows or candidates there are, nor on
which mix has computed a candidate's norm factor.  Bit for bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _mix(cands, inv, w, at=-1):
    from diff_gpt_b200 import ops

    h, rn = torch.empty_like(cands[0]), torch.empty_like(cands[0])
    new = torch.empty(cands[0].shape[0], device="cuda") if at >= 0 else None
    ops.depthmix_cached(cands, inv, w, h, rn, new, at)
    return h, rn, new


def _candidates(rows, C, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(C + n)
    base = torch.randn((rows, C), generator=g, device="cuda")
    return [(torch.roll(base, i, 0) * (1 + 0.3 * (i % 5))).to(dtype) for i in range(n)], (torch.randn(C, generator=g, device="cuda") * 0.2).to(dtype)


@pytest.mark.parametrize("C,n,dtype", [
    (256, 3, torch.bfloat16), (128, 5, torch.bfloat16), (40, 6, torch.bfloat16), (264, 4, torch.bfloat16), (512, 9, torch.bfloat16),
    (768, 13, torch.bfloat16), (64, 33, torch.bfloat16), (64, 3, torch.float32), (100, 7, torch.float32), (128, 4, torch.float32), (300, 5, torch.float32),
])
def test_many_rows_are_their_slices(C, n, dtype):
    """More candidates than L2 holds against slices that fit it."""
    rows = int(130e6 / (C * (2 if dtype == torch.bfloat16 else 4) * n)) | 1
    cands, w = _candidates(rows, C, n, dtype)
    inv, step = [None] * n, (rows + 7) // 8
    whole = _mix(cands, inv, w, 1)
    parts = [_mix([c[a : a + step] for c in cands], inv, w, 1) for a in range(0, rows, step)]
    for i in range(3):
        assert torch.equal(whole[i], torch.cat([p[i] for p in parts])), i


@pytest.mark.parametrize("C,dtype", [(256, torch.bfloat16), (120, torch.bfloat16), (64, torch.float32), (128, torch.float32)])
def test_factor_of_a_smaller_mix(C, dtype):
    """Two candidates fit L2 and leave the second one's factor; three do not, and use it."""
    rows = int(55e6 / (C * (2 if dtype == torch.bfloat16 else 4))) | 1
    cands, w = _candidates(rows, C, 3, dtype)
    factor = _mix(cands[:2], [None, None], w, 1)[2]
    for a, b in zip(_mix(cands, [None, factor, None], w)[:2], _mix(cands, [None] * 3, w)[:2]):
        assert torch.equal(a, b)
