"""Depth mix over more bytes than L2 holds (candidates fetched ahead, 16 lanes a row where it is short) against the same rows in
slices that take the kernel with a warp per row."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,n,dtype", [
    (256, 3, torch.bfloat16), (256, 1, torch.bfloat16), (128, 5, torch.bfloat16), (40, 6, torch.bfloat16), (264, 4, torch.bfloat16),
    (512, 9, torch.bfloat16), (768, 13, torch.bfloat16), (1000, 4, torch.bfloat16), (64, 33, torch.bfloat16), (64, 3, torch.float32),
    (100, 7, torch.float32), (300, 5, torch.float32), (512, 2, torch.float32),
])
def test_many_rows_equal_their_slices(C, n, dtype):
    """Sums of the two kernels differ in order only: the logit of a candidate by 2^-20 of its terms before it is rounded to the storage
    type, so by one step of it at most; that moves a weight by 2^-8 (bf16) of itself, and the result is rounded twice more."""
    from diff_gpt_b200 import ops

    size = 2 if dtype == torch.bfloat16 else 4
    rows = int(130e6 / (C * size * n)) | 1  # odd: the last pair of rows is half empty
    g = torch.Generator(device="cuda").manual_seed(C + n)
    base = torch.randn((rows, C), generator=g, device="cuda")
    cands = [(torch.roll(base, i, 0) * (1 + 0.3 * (i % 5))).to(dtype) for i in range(n)]
    w = (torch.randn(C, generator=g, device="cuda") * 0.2).to(dtype) if n > 1 else None
    inv = [None if i % 2 else torch.rand(rows, generator=g, device="cuda") + 0.5 for i in range(n)]
    if n == 1:
        inv = [None]
    at = 1 if n > 1 else -1

    def run(sl):
        m = cands[0][sl].shape[0]
        h, rn = (torch.full((m, C), float("nan"), dtype=dtype, device="cuda") for _ in range(2))
        new = torch.full((m,), float("nan"), device="cuda") if at >= 0 else None
        ops.depthmix_cached([c[sl] for c in cands], [None if v is None else v[sl] for v in inv], w, h, rn, new, at)
        return h, rn, new

    whole = run(slice(0, rows))
    step = (rows + 7) // 8
    parts = [run(slice(a, min(a + step, rows))) for a in range(0, rows, step)]
    for i in range(3):
        if whole[i] is None:
            continue
        a, b = whole[i].float(), torch.cat([p[i] for p in parts]).float()
        assert torch.isfinite(a).all()
        tol = 3 * 2.0**-8 if dtype == torch.bfloat16 and i < 2 else 2e-5
        scale = b.square().mean(-1, keepdim=True).sqrt() if i < 2 else b
        assert bool(((a - b).abs() <= tol * torch.maximum(b.abs(), scale)).all()), i
