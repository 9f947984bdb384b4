"""Which attention kernels run in front of draws: they round differently, so neither the number of rows nor that of prompts may choose between
them, and a job's tokens stay what they were."""

import pytest
import torch

from diff_gpt_b200 import GPT, TemperatureSampler, ops
from diff_gpt_b200.model.engine import DecodeRun

pytestmark = pytest.mark.gpu


def _model(C, H, L=2):
    torch.manual_seed(1)
    m = GPT(vocab_size=512, n_embd=C, block_size=1024, n_head=H, n_layer=L)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05)
    return m.to(torch.bfloat16).cuda().eval()


@pytest.mark.parametrize("C,H", [(128, 4), (256, 8), (512, 8), (768, 12)])
def test_the_shared_phase_runs_on_one_kernel(monkeypatch, C, H):
    """The phase over a prompt that 16 rows or more share: two query tiles a CTA, at every number of heads, rows and series."""
    seen, call = set(), ops.fmha_prefill
    monkeypatch.setattr(ops, "fmha_prefill", lambda *a, **kw: (seen.add(kw["impl"]) if kw.get("lse") is not None else None, call(*a, **kw))[1])
    model = _model(C, H)
    for S, N, P in ((1, 200, 300), (3, 33, 70), (1, 1200, 130)):
        ids = torch.randint(0, 512, (S, P), device="cuda", dtype=torch.int32)
        with torch.inference_mode():
            r = DecodeRun(model, ids, N, 3, TemperatureSampler(1.0), 0, None, use_graph=False)
            r.start()
            r.advance(3)
            r.check_status()
    assert seen == {4}
