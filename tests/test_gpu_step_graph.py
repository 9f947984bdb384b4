"""Single tokens through StepRunner (recorded launches) against the general path behind a cache of its own, bit for bit."""

import pytest
import torch

import delunex_cases
import kipolix_cases

pytestmark = pytest.mark.gpu


def _model(family, dtype):
    if family == "gpt":
        from diff_gpt_b200 import GPT

        torch.manual_seed(0)
        m = GPT(vocab_size=128, n_embd=96, block_size=2048, n_head=3, n_layer=3)
        for p in m.parameters():
            torch.nn.init.normal_(p, std=0.1)
        return m.to(dtype).cuda().eval(), 128
    cases = {"delunex": delunex_cases, "kipolix": kipolix_cases}[family]
    cfg = cases.CASES["wide"]
    return cases.build(cfg, 5, dtype)[0], cfg["vocab"]


def _plain(model, cache, ids):
    idx = torch.tensor([ids], device="cuda")
    return model.logits_at(idx, cache, torch.tensor([len(ids) - 1], device="cuda")).float().clone()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("family", ["gpt", "delunex", "kipolix"])
def test_recorded_steps_equal_the_general_path(family, dtype):
    """From the first token over 1200 tokens: every count of key splits, portions in between (which swap the state buffer), a
    grown or moved cache, weights changed on the way, and a second request that takes the cache over."""
    from diff_gpt_b200 import StepRunner

    model, V = _model(family, dtype)
    runner = StepRunner(model)
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, V, (1300,), generator=g).tolist()
    for n_tokens, portions in ((1300, {5: 3, 40: 120, 300: 40, 900: 150}), (30, {0: 7})):
        cache = model.new_cache()
        cache.reset()
        at, part = 0, []
        with torch.inference_mode():
            while at < n_tokens:
                n = min(portions.get(at, 1), n_tokens - at)
                got = runner.step("r", ids[at : at + n], [n - 1])
                part.append(torch.equal(got, _plain(model, cache, ids[at : at + n])))
                at += n
                if at == 700:
                    w = model.token_embedding_table.weight if family == "gpt" else model.embed
                    w.mul_(1.25)
        assert all(part), [i for i, ok in enumerate(part) if not ok][:5]
        assert any(one.graph is not None for one in runner._single.values())
        runner.finish("r")
    assert len(runner._free) == 1 and len(runner._single) <= 2


@pytest.mark.parametrize("family,dtype", [("gpt", torch.float32), ("gpt", torch.bfloat16), ("kipolix", torch.bfloat16)])
def test_requests_on_their_own_streams(family, dtype):
    """Two requests stepped from two streams give what they give alone.  A GPT's step returns with its work pending: nothing waits on the
    host from the prompts to the end, while one request passes 512 keys (another plan and recording) and the other outgrows its
    cache; results are copied out on the callers' streams and their memory used again.  (The other models read a status after every
    step, which makes the host wait for it.)"""
    from diff_gpt_b200 import StepRunner

    model, V = _model(family, dtype)
    runner = StepRunner(model)
    first = {0: 500, 1: 2038} if family == "gpt" else {0: 1, 1: 1}
    ids = {k: torch.randint(0, V, (first[k] + 60,), generator=torch.Generator().manual_seed(k)).tolist() for k in range(2)}
    want = {}
    for k, t in ids.items():
        cache = model.new_cache()
        cache.reset()
        with torch.inference_mode():
            want[k] = torch.cat([_plain(model, cache, t[: first[k]])] + [_plain(model, cache, [x]) for x in t[first[k] :]])
    streams = [torch.cuda.Stream() for _ in ids]
    got = {k: torch.zeros_like(want[k]) for k in ids}
    torch.cuda.synchronize()
    for k in ids:
        with torch.cuda.stream(streams[k]):
            got[k][:1].copy_(runner.step(k, ids[k][: first[k]], [first[k] - 1]))
    for i in range(60):
        for k in ids:
            with torch.cuda.stream(streams[k]):
                got[k][i + 1 : i + 2].copy_(runner.step(k, [ids[k][first[k] + i]], [0]))
                torch.full((1, V), float("nan"), device="cuda")  # in the place of the result just dropped
    torch.cuda.synchronize()
    for k in ids:
        assert torch.equal(got[k], want[k]), k


@pytest.mark.parametrize("family,dtype", [("gpt", torch.float32), ("gpt", torch.bfloat16), ("delunex", torch.bfloat16), ("kipolix", torch.bfloat16)])
def test_parameters_that_are_views_off_16_bytes(family, dtype):
    """Layer weights four or two bytes off a 16-byte boundary (views into one buffer) give what aligned ones give, up to the order of
    the sums: single tokens and short prompts took any alignment before the kernels for few rows."""
    model, V = _model(family, dtype)
    ids = torch.randint(0, V, (1, 12), generator=torch.Generator().manual_seed(3)).cuda()

    def run():
        cache = model.new_cache()
        cache.reset()
        rows = torch.tensor([0], device="cuda")
        with torch.inference_mode():
            first = model.logits_at(ids[:, :11], cache, torch.tensor([10], device="cuda")).float().clone()
            return torch.cat([first, model.logits_at(ids[:, 11:], cache, rows).float()])

    want = run()
    table = model.token_embedding_table.weight if family == "gpt" else None
    for name, p in model.named_parameters():
        if p.dim() == 2 and p.shape[0] > 1 and p is not table and name not in ("embed", "head", "bigram"):
            flat = torch.empty(p.numel() + 1, dtype=dtype, device="cuda")
            flat[1:].copy_(p.detach().reshape(-1))
            p.data = flat[1:].view(p.shape)
    got = run()
    assert (got - want).abs().max().item() <= (1e-5 if dtype == torch.float32 else 3e-2) * want.abs().max().item()
