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


@pytest.mark.parametrize("P", [640, 768])
@pytest.mark.parametrize("C,H", [(256, 8), (512, 8)])
def test_prompts_prefilled_in_groups(C, H, P):
    """Ranks that share the prefill of a job's prompts hold what one rank would."""
    model = _model(C, H)
    ids = torch.randint(0, 512, (16, P), generator=torch.Generator().manual_seed(P)).to(torch.int32).cuda()

    def logits0(rows):
        with torch.inference_mode():
            return DecodeRun(model, rows.contiguous(), 1, 2, TemperatureSampler(1.0), 0, None, whole_job=False).logits0.clone()

    whole = logits0(ids)
    assert torch.equal(whole, torch.cat([logits0(ids[:8]), logits0(ids[8:])]))


@pytest.mark.parametrize("B,H,T", [(1, 8, 64), (3, 8, 200), (24, 8, 256), (16, 12, 512), (64, 4, 700)])
def test_prompts_in_pages_keep_their_kernel(B, H, T):
    """Heads of 32 in pages: the tcgen05 kernels, as before dense sequences had a kernel of their own."""
    D, pt = 32, 64
    C, n = H * D, -(-T // pt)
    g = torch.Generator(device="cuda").manual_seed(T)
    pool = torch.randn((B * n, 2, H, pt, D), generator=g, device="cuda").bfloat16()
    table = torch.randperm(B * n, generator=g, device="cuda").to(torch.int32).view(B, n).contiguous()
    q = torch.randn((B * T, C), generator=g, device="cuda").bfloat16()
    lay = ops.kv_layout(pool[0, 0], pool[0, 1], 2 * H * pt * D, pt * D, pt, table, pool.shape[0])
    status, outs = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    for impl in (0, 2, 3):
        y = torch.empty_like(q)
        ops.fmha_prefill(q, lay, y, B=B, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C, o_batch_stride=T * C, o_row_stride=C, kv_len_all=T,
                         causal=True, status=status, impl=impl)
        outs.append(y)
    assert status.item() == 0 and (torch.equal(outs[0], outs[1]) or torch.equal(outs[0], outs[2]))


@pytest.mark.parametrize("causal", [True, False])
def test_a_length_per_dense_sequence(causal):
    """Dense keys of heads of 32, products in registers: a length per sequence, one of none at all; error against float64 as in test_gpu_fmha_mma."""
    B, H, D, T = 40, 5, 32, 320
    C = H * D
    g = torch.Generator(device="cuda").manual_seed(4)
    kv = torch.randn((2, B, H, T, D), generator=g, device="cuda").bfloat16()
    kv_len = torch.randint(1, T + 1, (B,), generator=g, device="cuda").to(torch.int32)
    kv_len[0], kv_len[1] = 0, T
    q, y = torch.randn((B * T, C), generator=g, device="cuda").bfloat16(), torch.full((B * T, C), float("nan"), device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.fmha_prefill(q, ops.kv_layout(kv[0], kv[1], H * T * D, T * D, T), y, B=B, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C,
                     o_batch_stride=T * C, o_row_stride=C, kv_len=kv_len, causal=causal, status=status)
    s = q.double().view(B, T, H, D).transpose(1, 2) @ kv[0].double().transpose(-1, -2) * D**-0.5
    j = torch.arange(T, device="cuda")
    seen = (j[None] < kv_len[:, None])[:, None, None].expand(B, 1, T, T)
    if causal:
        seen = seen & (j[None] <= j[:, None])
    p = torch.softmax(s.masked_fill(~seen, float("-inf")), -1).nan_to_num(0.0)
    ref = (p @ kv[1].double()).transpose(1, 2).reshape(B * T, C)
    assert (y.double() - ref).norm() <= 4e-3 * ref.norm() and status.item() == 0 and bool((y[:T] == 0).all())
