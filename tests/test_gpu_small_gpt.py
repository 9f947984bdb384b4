"""A small fp32 GPT's forwards and decode steps as one launch (dgpt_small_gpt) against the launches of the general path."""

import pytest
import torch

from diff_gpt_b200 import GPT, NucleusSampler, StepRunner, TemperatureSampler
from diff_gpt_b200.model import gpt as gpt_module
from diff_gpt_b200.model.engine import DecodeRun

pytestmark = pytest.mark.gpu

# fp32 on both sides, sums of at most 256 terms over at most 8 layers, in two orders: 2e-6 measured, and each side is as far from 64 bits
REL = 1e-5


def _model(C, H, L, V, per_block=1, cap=15.0):
    g = torch.Generator(device="cuda").manual_seed(C + H + L + V)
    with torch.device("cuda"):
        m = GPT(vocab_size=V, n_embd=C, n_head=H, n_layer=L, block_size=512, attn_res_layers_per_block=per_block, logit_softcap=cap,
                pad_vocab_size_to=4)
    m = m.cuda().eval()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * 1.2 / C**0.5)
    return m


def _both(monkeypatch, f):
    """f() on one launch per forward, and on the general path."""
    with monkeypatch.context() as mp:
        mp.setattr(gpt_module, "whole_f32", lambda C, H, L, V, n_seq, T, keys: gpt_module.ops.small_gpt_supported(C, H, L, V, keys))
        one = f()
    with monkeypatch.context() as mp:
        mp.setattr(gpt_module, "whole_f32", lambda *a: False)
        return one, f()


def _close(a, b):
    assert (a - b).norm() <= REL * b.norm()


SHAPES = [(32, 4, 1, 64, 1), (32, 1, 3, 260, 2), (64, 4, 2, 256, 1), (64, 8, 3, 1024, 3), (64, 2, 2, 100, 1), (128, 16, 2, 36, 1), (128, 4, 8, 512, 4)]


@pytest.mark.parametrize("C,H,L,V,per_block", SHAPES)
@pytest.mark.parametrize("B,T", [(1, 1), (1, 16), (1, 17), (2, 129), (40, 7), (3, 300)])
def test_forward(monkeypatch, C, H, L, V, per_block, B, T):
    m = _model(C, H, L, V, per_block)
    idx = torch.randint(0, V, (B, T), device="cuda")
    _close(*_both(monkeypatch, lambda: m(idx)[0]))


# rows around the numbers where a CTA takes 1, 2, 4 or 8 of them; prompts around page edges
@pytest.mark.parametrize("C,H,L,V,per_block", [SHAPES[0], SHAPES[2], SHAPES[6]])
@pytest.mark.parametrize("S,N,P", [(1, 1, 1), (2, 3, 64), (1, 149, 65), (3, 99, 130), (1, 593, 40)])
@pytest.mark.parametrize("top_p", [1.0, 0.8])
def test_decode(monkeypatch, C, H, L, V, per_block, S, N, P, top_p):
    m, G = _model(C, H, L, V, per_block), 7
    ids = torch.randint(0, V, (S, P + G), device="cuda")
    sampler = NucleusSampler(top_p, TemperatureSampler(0.7)) if top_p < 1 else TemperatureSampler(1.0)
    force = [r[:-1] + [None] for r in ids[:, P:].tolist()]  # given tokens: the last logits are a function of the inputs

    def run():
        with torch.inference_mode():
            r = DecodeRun(m, ids[:, :P].to(torch.int32).contiguous(), N, G, sampler, 3, force)
            r.start()
            r.advance(2)
            r.advance(G)
            r.check_status()
            return r.logits.clone(), r.tokens_so_far().clone()

    (za, ta), (zb, tb) = _both(monkeypatch, run)
    _close(za, zb)
    assert torch.equal(ta[:, :-1], tb[:, :-1])
    assert (ta[:, -1] != tb[:, -1]).float().mean() <= 0.01  # a draw between two tokens may fall to the other


@pytest.mark.parametrize("temperature", [0.0, 0.6, 1.0])
@pytest.mark.parametrize("V", [252, 512, 1024])
def test_free_draws(monkeypatch, V, temperature):
    m = _model(64, 4, 2, V)
    prompt = torch.randint(0, V, (1, 30), device="cuda").to(torch.int32)

    def run():
        with torch.inference_mode():
            r = DecodeRun(m, prompt, 200, 6, TemperatureSampler(temperature), 11, None)
            r.start()
            r.advance(6)
            return r.tokens_so_far().clone()

    a, b = _both(monkeypatch, run)
    assert (a != b).any(1).float().mean() <= 0.01


def test_steps(monkeypatch):
    m = _model(64, 4, 2, 256)
    tokens = torch.randint(0, 256, (320,)).tolist()

    def run():
        r = StepRunner(m)
        out = [r.step(0, tokens[:250], [0, 249])] + [r.step(0, [t], [0]) for t in tokens[250:260]]  # past the plan's 256 keys
        out.append(r.step(0, tokens[260:], [59]))
        return torch.cat(out)

    _close(*_both(monkeypatch, run))


def test_out_of_range_is_reported(monkeypatch):
    m = _model(32, 4, 1, 64)
    prompt = torch.randint(0, 64, (1, 4), device="cuda").to(torch.int32)
    with torch.inference_mode():
        r = DecodeRun(m, prompt, 5, 6, TemperatureSampler(1.0), 0, None)
        assert r.plan.whole
        r.start()
        r.bind.pos0 += m.freqs_cis.shape[0]
        r.advance(1)
        with pytest.raises(RuntimeError, match="status 1"):
            r.check_status()


@pytest.mark.parametrize("R", [3, 200, 700])  # one, two and eight rows a CTA
@pytest.mark.parametrize("slot,start,length,keys", [(20, 0, 21, 21), (20, 0, 20, 21), (20, 0, 12, 40), (5, 0, 20, 20), (9, 4, 15, 32)])
def test_tokens_whose_own_key_is_not_the_last(R, slot, start, length, keys):
    """slot: where the token's key goes; start, length: the keys that it sees, its own the last of them, in between or not among them."""
    from diff_gpt_b200.model.gpt import ForwardPlan, KvBinding
    from diff_gpt_b200.model.kv_cache import KVCache

    m = _model(32, 4, 3, 64)
    g = torch.Generator(device="cuda").manual_seed(R + slot)
    ids = torch.randint(0, 64, (R,), generator=g, device="cuda", dtype=torch.int32)
    storage = torch.randn((3, 2, R, 4, 48, 8), generator=g, device="cuda")
    i32 = lambda x: torch.full((R,), x, dtype=torch.int32, device="cuda")  # noqa: E731

    def run(whole):
        cache = KVCache(R, 4, 48, 8, 3)
        cache.kv_cache = storage.clone()
        bind = KvBinding(layouts=[cache.layer_layout(i) for i in range(3)], pos0=i32(20), slot0=i32(slot), decode=True, len0=i32(0), start1=i32(start),
                         len1=i32(length), n_splits=1)
        with torch.inference_mode():
            plan = ForwardPlan(m, R, 1, keys=keys if whole else None)
            assert plan.whole == whole
            return plan.run(ids, bind).clone(), cache.kv_cache, int(plan.status)

    (za, ca, sa), (zb, cb, sb) = run(True), run(False)
    _close(za, zb)
    _close(ca, cb)
    assert sa == sb == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("temperature,V", [(0.0, 256), (1.0, 256), (0.7, 512)])
def test_numbers_that_are_none(monkeypatch, bad, temperature, V):
    """A token whose vector is not finite: the logits of every token that sees it are not either, and the draws from such rows go by one rule."""
    m = _model(64, 4, 2, V, cap=0.0)
    with torch.no_grad():
        m.token_embedding_table.weight[5] = bad
    idx = torch.randint(6, V, (3, 40), device="cuda")
    idx[1, 17] = 5

    one, plain = (x.isfinite() for x in _both(monkeypatch, lambda: m(idx)[0]))
    assert not bool(one[1, 17:].any()) and bool(one[1, :17, 6:].all()) and bool(one[::2, :, 6:].all())
    assert not bool((plain & ~one).any())  # (the general path multiplies what a row does not see by 0, and so loses more rows)

    def draws():
        with torch.inference_mode():
            r = DecodeRun(m, idx[:, :30].to(torch.int32).contiguous(), 20, 5, TemperatureSampler(temperature), 11, None)
            r.start()
            r.advance(5)
            return r.tokens_so_far().clone()

    a, b = _both(monkeypatch, draws)
    assert torch.equal(a, b)


def test_a_late_status_is_raised(monkeypatch):
    """Nobody waits for a forward or a recorded token: what its kernel reports is raised by the next call, and by `finish` at the latest.  (Made by
    positions beyond the table, which the kernel clamps; a copy of the model has a word of its own.)"""
    import copy

    m = _model(32, 4, 1, 64)
    idx = torch.randint(0, 64, (1, 8), device="cuda")
    m(idx)
    torch.cuda.synchronize()
    m(idx)
    other, table = copy.deepcopy(m), m.freqs_cis.shape[0]
    real = gpt_module.ops.small_gpt

    def far(model, kv, stride, ids, pos0, *a, **kw):
        real(model, kv, stride, ids, pos0 + table, *a, **kw)

    with monkeypatch.context() as mp:
        mp.setattr(gpt_module.ops, "small_gpt", far)
        m(idx)
    torch.cuda.synchronize()
    other(idx)
    with pytest.raises(RuntimeError, match="status 1"):
        m(idx)
    m(idx)  # raised once
    r = StepRunner(m)
    r.step("a", [1, 2, 3], [2])
    for _ in range(3):
        r.step("a", [4], [0])
    with monkeypatch.context() as mp:
        mp.setattr(gpt_module.ops, "small_gpt", far)
        r.step("b", [1, 2], [1])
    with pytest.raises(RuntimeError, match="status 1"):
        r.finish("b")
    r.step("a", [5], [0])
    r.finish("a")
    torch.cuda.synchronize()
