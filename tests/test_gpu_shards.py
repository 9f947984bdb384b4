"""A shard of a bf16 batch has the logits, bit for bit, and so the tokens, that its rows have in the whole batch; down to one row."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(C, H, V):
    from diff_gpt_b200 import GPT

    torch.manual_seed(0)
    m = GPT(vocab_size=V, n_embd=C, block_size=1024, n_head=H, n_layer=2)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05)
    return m.to(torch.bfloat16).cuda().eval()


@pytest.mark.parametrize("C,H,V", [(256, 8, 512), (128, 2, 256), (64, 4, 256)])  # heads of 32 and 64, and of 16 (warp-level kernel)
@pytest.mark.parametrize("P,N,n,overlap", [(100, 40, 1, True), (100, 40, 1, False), (300, 40, 2, True), (700, 300, 20, False), (100, 8, 1, True), (90, 8, 2, True)])
def test_logits_of_a_shard(C, H, V, P, N, n, overlap):
    from diff_gpt_b200 import NucleusSampler, TemperatureSampler
    from diff_gpt_b200.model.engine import DecodeRun

    model, G = _model(C, H, V), 6
    prompts = [torch.randint(0, V, (P,), generator=torch.Generator().manual_seed(s)).tolist() for s in range(2)]
    force = [[(7 * g + s) % 200 for g in range(G - 1)] + [None] for s in range(2)]

    def run(rows, prompts, force, sampler):
        with torch.inference_mode():
            r = DecodeRun(model, prompts, rows, G, sampler, 42, force, shared_prefix=N >= 16, overlap_prefix=overlap, fused_head=False,
                          whole_job=False)
            r.start()
            r.advance(G)
            r.check_status()
            return r.logits0.clone(), r.logits.view(len(prompts), rows, -1).clone()

    for sampler in (TemperatureSampler(1.0), NucleusSampler(0.9, TemperatureSampler(1.0))):
        whole = run(N, prompts[:1], force[:1], sampler)
        part = run(n, prompts[:1], force[:1], sampler)
        assert torch.equal(whole[0], part[0]) and torch.equal(whole[1][:, :n], part[1])


@pytest.mark.parametrize("N,shards", [(40, 40), (8, 8), (24, 12)])
def test_tokens_of_shards(N, shards):
    from diff_gpt_b200 import Engine, NucleusSampler, TemperatureSampler

    model = _model(256, 8, 512)
    prompt = torch.randint(0, 512, (120,), generator=torch.Generator().manual_seed(5)).tolist()
    for sampler in (TemperatureSampler(1.0), NucleusSampler(0.9, TemperatureSampler(1.0))):
        whole, _ = Engine(model).generate_many([prompt], N, 30, sampler, seed=3)
        n = N // shards
        for i in range(0, N, 4 * n):
            part, _ = Engine(model).generate_many([prompt], n, 30, sampler, seed=3, traj_offset=i, shared_prefix=N >= 16)
            assert torch.equal(part, whole[:, i : i + n]), i


def test_tiles_at_any_number_of_rows():
    """dgpt_linear with `tiles`: one and two rows as they come out of 300."""
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(2)
    a, w = torch.randn(300, 520, generator=g, device="cuda").bfloat16(), torch.randn(1040, 520, generator=g, device="cuda").bfloat16()
    whole = torch.empty(300, 1040, dtype=torch.bfloat16, device="cuda")
    ops.linear(a, w, whole)
    for M in (1, 2, 3):
        out = torch.empty(M, 1040, dtype=torch.bfloat16, device="cuda")
        ops.linear(a[:M], w, out, tiles=True)
        assert torch.equal(out, whole[:M])


def _configured(family):
    if family == "delunex":
        from delunex_cases import build, config, mixer

        layers = [(mixer(16, 64, 64, 128, 200), 512), (mixer(16, 64, 64, 128, 90, kv_from=0), 512)]
        return build(config(256, 512, 3, layers), 3, torch.bfloat16)[0]
    from kipolix_cases import attention, build, config

    return build(config(256, 512, [(attention(16, 4, 64, 64, 200, 4), 512), (attention(16, 2, 64, 64, 90, 0), 512)]), 3, torch.bfloat16)[0]


@pytest.mark.parametrize("family", ["delunex", "kipolix"])
@pytest.mark.parametrize("P,N,n", [(300, 1024, 256), (40, 640, 320)])
def test_a_shard_of_rows_behind_one_prompt(family, P, N, n):
    """The number of rows chooses how many of them the attention takes together, which may not show in any of them.  (Numbers of rows for
    which the products run on the same kernels.)"""
    from diff_gpt_b200 import Engine, TemperatureSampler
    from diff_gpt_b200.model.engine import DecodeRun

    model, G = _configured(family), 40
    prompt = torch.randint(0, 512, (P,), generator=torch.Generator().manual_seed(P)).tolist()
    force = [[(7 * g) % 500 for g in range(G - 1)] + [None]]

    def logits(rows):
        with torch.inference_mode():
            r = DecodeRun(model, [prompt], rows, G, TemperatureSampler(1.0), 42, force, fused_head=False, whole_job=False)
            r.start()
            r.advance(G)
            r.check_status()
            return r.logits.clone()

    assert torch.equal(logits(N)[:n], logits(n))
    whole, _ = Engine(model).generate_many([prompt], N, 30, TemperatureSampler(1.0), seed=3)
    for i in range(0, N, 2 * n):
        part, _ = Engine(model).generate_many([prompt], n, 30, TemperatureSampler(1.0), seed=3, traj_offset=i)
        assert torch.equal(part, whole[:, i : i + n]), i
