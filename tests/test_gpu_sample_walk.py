"""Inverse-CDF draws at the seams between the lanes' (threads') shares of a row: millions of uniforms through one row of logits against a
float64 walk with the same uniforms.  A target that fp32 sums put between two shares belongs to a token beside the seam."""

import numpy as np
import pytest
import torch

from oracle import ref_decode

pytestmark = pytest.mark.gpu


def _uniforms(seed: int, n: int, attempt: int) -> np.ndarray:
    """Philox4x32-10 of counters (row, 0, 0, attempt): the first word's upper 24 bits, as the kernels use them."""
    c = [np.arange(n, dtype=np.uint64), *(np.full(n, v, dtype=np.uint64) for v in (0, 0, attempt))]
    k0, k1, low = np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32), np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & low]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & low, (k1 + np.uint64(0xBB67AE85)) & low
    return (c[0] >> np.uint64(8)).astype(np.float64) / 16777216.0


@pytest.mark.parametrize("V,log2_rows,scale,T,top_p", [
    (256, 23, 0.16, 1.0, 1.0),   # a warp per row
    (1000, 22, 1.0, 0.8, 1.0),   # the same, temperature applied on the way, a short last share
    (256, 23, 1.0, 4.0, 0.3),    # the same, walk over a nucleus after eight rejected draws
    (12300, 22, 0.5, 1.0, 1.0),  # a CTA per row
])
def test_every_target_ends_beside_its_place(V, log2_rows, scale, T, top_p):
    """The sums are fp32, so a token next to the exact one is allowed (its edge lies within rounding), any other is not."""
    from diff_gpt_b200 import ops

    R, seed = 1 << log2_rows, 0x2468_1357
    logits = torch.randn(1, V, generator=torch.Generator().manual_seed(V)) * scale
    out = torch.empty(R, dtype=torch.int32, device="cuda")
    ops.sample(logits.cuda(), out, R=R, row_stride=0, temperature=T, top_p=top_p, seed=seed)
    got = out.cpu().numpy()
    z = logits[0].double()
    w = torch.exp((z - z.max()) / T).numpy()
    rows = np.arange(R)
    kept = np.arange(V)
    attempt = 0
    if top_p < 1:
        mask = ref_decode.nucleus_mask(logits, top_p)[0].numpy()
        near = mask | np.roll(mask, 1) | np.roll(mask, -1)
        cdf = np.cumsum(w) / w.sum()
        for attempt in range(8):  # rows whose draws over all tokens fall clear of the nucleus every time
            cand = np.searchsorted(cdf, _uniforms(seed, R, attempt)[rows], side="right").clip(max=V - 1)
            rows = rows[~near[cand]]
        kept, attempt = np.nonzero(mask)[0], 8
        assert rows.size > R // 20 and mask[got].all()
    cdf = np.cumsum(w[kept]) / w[kept].sum()
    want = np.searchsorted(cdf, _uniforms(seed, R, attempt)[rows], side="right").clip(max=kept.size - 1)
    off = np.abs(np.searchsorted(kept, got[rows]) - want)
    far = np.nonzero(off > 1)[0]
    assert far.size == 0, (far.size, rows[far[:5]].tolist(), got[rows[far[:5]]].tolist(), kept[want[far[:5]]].tolist())
    assert (off == 1).mean() < 1e-3
