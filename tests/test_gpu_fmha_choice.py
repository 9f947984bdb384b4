"""Every choice of prefill-attention kernel that a caller of the engine can name gives the same prompt."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["gpt", "delunex", "kipolix"])
@pytest.mark.parametrize("impl", [1, 2, 3, 4])
def test_generate_many_takes_every_kernel(family, impl):
    """Against the library's own choice: bf16 logits of two kernels differ by their order of sums (2e-2 of the largest, as elsewhere)."""
    import delunex_cases
    import kipolix_cases
    from diff_gpt_b200 import GPT, Engine, TemperatureSampler

    if family == "gpt":
        torch.manual_seed(0)
        model = GPT(vocab_size=128, n_embd=128, block_size=1024, n_head=2, n_layer=2)
        for p in model.parameters():
            torch.nn.init.normal_(p, std=0.1)
        model, V = model.to(torch.bfloat16).cuda().eval(), 128
    else:
        cases = {"delunex": delunex_cases, "kipolix": kipolix_cases}[family]
        model, V = cases.build(cases.CASES["wide"], 5, torch.bfloat16)[0], cases.CASES["wide"]["vocab"]
    prompt = torch.randint(0, V, (300,), generator=torch.Generator().manual_seed(2)).tolist()
    logits = []
    for choice in (0, impl):
        engine = Engine(model)
        toks, _ = engine.generate_many([prompt], 2, 3, TemperatureSampler(0.0), fmha_impl=choice)
        assert toks.shape == (1, 2, 3)
        logits.append(engine._run.logits0.float())
    assert (logits[1] - logits[0]).abs().max().item() <= 2e-2 * logits[0].abs().max().item()
