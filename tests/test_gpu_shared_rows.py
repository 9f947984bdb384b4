"""Decode attention over cached rows where several sequences share a prompt's pages: rows taken together in one item."""

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [  # share, prompts, prompt keys, own keys, window, keep, page_tokens, splits
    (4, 3, 300, 33, 0, 0, 64, 1),     # two rows' own keys in one tile
    (5, 2, 130, 65, 100, 3, 64, 1),   # a set that is not full; own keys beyond half a tile; the window starts in the prompt
    (3, 2, 40, 200, 90, 2, 16, 1),    # the window has left the prompt, whose kept keys are still seen
    (7, 2, 3, 70, 20, 9, 32, 1),      # kept keys in the prompt and behind it
    (2, 3, 1, 1, 0, 0, 8, 1),         # the fewest keys
    (9, 2, 257, 64, 0, 5, 64, 3),     # splits, some of which hold a part of the rows only
    (33, 1, 500, 150, 400, 1, 128, 2),
]


def plain(q, k, v, gate, seen, scale):
    """float64 of q [H, dk], k [n, H, dk], v [n, H, dv], and sum_j p_j |v_j|."""
    s = torch.einsum("hd,nhd->hn", q, k) * scale
    p = torch.softmax(s.masked_fill(~seen, float("-inf")), dim=-1)
    g = 1.0 if gate is None else torch.sigmoid(gate)[:, None]
    return torch.einsum("hn,nhd->hd", p, v) * g, torch.einsum("hn,nhd->hd", p, v.abs()) * g


@pytest.mark.parametrize("H,G,dk", [(16, 0, 512), (16, 0, 64), (8, 0, 136), (16, 4, 128), (16, 8, 64), (4, 4, 96), (32, 1, 64)])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_rows_of_one_prompt_together(case, H, G, dk):
    """G = 0: latents.  Every number of rows together, the chosen one, and each row by itself, against float64."""
    from diff_gpt_b200 import ops

    share, prompts, n_prompt, n_own, window, keep, pt, splits = case
    latents = G == 0
    keep, groups = (0, 1) if latents else (keep, G)
    width = dk if latents else 2 * G * dk
    R, per = share * prompts, H // groups
    g = torch.Generator().manual_seed(R + H + dk)
    pp, op = -(-n_prompt // pt), -(-n_own // pt)
    n_pages = prompts * pp + R * op
    pool = torch.full((n_pages, pt, width), float("nan"))
    perm = torch.randperm(n_pages, generator=g).int()
    table = torch.cat([perm[: prompts * pp].view(prompts, pp).repeat_interleave(share, 0), perm[prompts * pp :].view(R, op)], 1)
    rows = torch.randn(prompts, n_prompt, width, generator=g).bfloat16()
    own = torch.randn(R, n_own, width, generator=g).bfloat16()
    for r in range(R):
        for t, x in enumerate(rows[r // share]):
            pool[table[r, t // pt], t % pt] = x.float()
        for t, x in enumerate(own[r]):
            pool[table[r, pp + t // pt], t % pt] = x.float()
    # slots between a page's last written key and its end hold NaN: they may not reach a result
    store, table = pool.bfloat16().cuda(), table.contiguous().cuda()
    q = (2 * torch.randn(R, H * dk, generator=g)).bfloat16()
    gate = torch.randn(R, H, generator=g).bfloat16()
    scale, n = dk**-0.5, n_prompt + n_own
    j = torch.arange(n)
    seen = (j < keep) | (j >= n - window) if window else torch.ones(n, dtype=torch.bool)
    want, size = [], []
    for r in range(R):
        x = torch.cat([rows[r // share], own[r]]).double()
        k = x.view(n, groups, dk) if latents else x[:, : G * dk].reshape(n, G, dk)
        v = k if latents else x[:, G * dk :].reshape(n, G, dk)
        o, a = plain(q[r].double().view(H, dk), k.repeat_interleave(per, 1), v.repeat_interleave(per, 1), gate[r].double(), seen, scale)
        want.append(o.reshape(-1))
        size.append(a.reshape(-1))
    want, size = torch.stack(want), torch.stack(size)
    i32 = lambda x: torch.full((R,), x, dtype=torch.int32, device="cuda")  # noqa: E731
    step = torch.full((1,), n_own - 1, dtype=torch.int32, device="cuda")
    lay = ops.kv_layout(store, store, store.stride(0), 0, pt, table, n_pages)
    together = [0, 1] + [t for t in (2, 4, 8, 16, 32, 64) if per & (per - 1) == 0 and 16 <= per * t <= 64]
    for t in together:
        out = torch.full((R, H * dk), float("nan"), dtype=torch.bfloat16, device="cuda")
        ws = torch.empty(max(4, ops.latent_attn_workspace_bytes(R, H, dk, splits) // 4), device="cuda") if splits > 1 else None
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = dict(n_seq=R, T=1, H=H, window=window, scale=scale, gate=gate.cuda(), workspace=ws, n_splits=splits, share=share, together=t,
                  prompt_keys=n_prompt, own_keys=n_own, status=st)
        args = (q.cuda(), lay, i32(n_prompt), i32(pp * pt), i32(1), step, out)
        if latents:
            ops.latent_attn(*args, r=dk, **kw)
        else:
            ops.grouped_attn(*args, row_width=width, v_col=G * dk, G=G, dk=dk, dv=dk, keep_first=keep, **kw)
        assert int(st) == 0
        # a probability and the result are rounded to bf16 once each (eight significant bits: 2^-8), sums are fp32
        bound = 2**-8 * (size + want.abs()) * 1.02 + 1e-5
        assert bool(((out.double().cpu() - want).abs() <= bound).all()), (t, float(((out.double().cpu() - want).abs() / bound).max()))


def test_a_prompt_is_shared_by_whole_runs_of_rows():
    from diff_gpt_b200 import ops
    from diff_gpt_b200._lib import DgptError

    x = torch.zeros(3, 16 * 64, dtype=torch.bfloat16, device="cuda")
    store, one = torch.zeros(3, 64, 64, dtype=torch.bfloat16, device="cuda"), torch.ones(3, dtype=torch.int32, device="cuda")
    lay = ops.kv_layout(store, store, store.stride(0), 0, 64)
    for kw in (dict(share=2), dict(share=0), dict(share=3, together=3), dict(share=3, together=8)):
        with pytest.raises(DgptError):
            ops.latent_attn(x, lay, None, one, one, None, x, n_seq=3, T=1, H=16, r=64, window=0, scale=1.0, **kw)


@pytest.mark.parametrize("H,G,dk", [(16, 0, 512), (16, 0, 64), (8, 0, 136), (32, 0, 128), (16, 4, 128), (16, 8, 64), (32, 4, 96), (32, 1, 64), (64, 2, 64)])
@pytest.mark.parametrize("case", CASES + [(6, 2, 200, 64, 0, 0, 32, 2), (8, 3, 130, 129, 0, 3, 64, 3), (31, 1, 260, 30, 120, 2, 16, 3)],
                         ids=lambda c: "x".join(map(str, c)))
def test_a_row_has_the_bits_that_it_gets_by_itself(case, H, G, dk):
    """However many rows are taken together, with splits and without: the order of a row's sums is its own."""
    from diff_gpt_b200 import ops

    share, prompts, n_prompt, n_own, window, keep, pt, splits = case
    keep, groups = (0, 1) if G == 0 else (keep, G)
    width = dk if G == 0 else 2 * G * dk
    R, per = share * prompts, H // groups
    g = torch.Generator(device="cuda").manual_seed(R + H + dk)
    pp, op = -(-n_prompt // pt), -(-n_own // pt)
    n_pages = prompts * pp + R * op
    store = torch.randn((n_pages, pt, width), generator=g, device="cuda").bfloat16()
    perm = torch.randperm(n_pages, generator=g, device="cuda").int()
    table = torch.cat([perm[: prompts * pp].view(prompts, pp).repeat_interleave(share, 0), perm[prompts * pp :].view(R, op)], 1).contiguous()
    # some rows' largest scores come late in the prompt or among their own keys, by more than the 2^8 that moves a reference
    q = torch.randn((R, H * dk), generator=g, device="cuda") * torch.rand((R, 1), generator=g, device="cuda") * 12
    q, gate = q.bfloat16(), torch.randn((R, H), generator=g, device="cuda").bfloat16()
    i32 = lambda x: torch.full((R,), x, dtype=torch.int32, device="cuda")  # noqa: E731
    step = torch.full((1,), n_own - 1, dtype=torch.int32, device="cuda")
    lay = ops.kv_layout(store, store, store.stride(0), 0, pt, table, n_pages)

    def run(together):
        out = torch.full((R, H * dk), float("nan"), dtype=torch.bfloat16, device="cuda")
        ws = torch.empty(max(4, ops.latent_attn_workspace_bytes(R, H, dk, splits) // 4), device="cuda").fill_(float("nan")) if splits > 1 else None
        kw = dict(n_seq=R, T=1, H=H, window=window, scale=dk**-0.5, gate=gate, workspace=ws, n_splits=splits, share=share, together=together,
                  prompt_keys=5000, own_keys=1)  # (so that a number is chosen which shares)
        args = (q, lay, i32(n_prompt), i32(pp * pt), i32(1), step, out)
        if G == 0:
            ops.latent_attn(*args, r=dk, **kw)
        else:
            ops.grouped_attn(*args, row_width=width, v_col=G * dk, G=G, dk=dk, dv=dk, keep_first=keep, **kw)
        return out

    counts = [0] + [t for t in (2, 4, 8, 16) if 16 <= per * t <= 64]
    want = run(1)
    assert bool(torch.isfinite(want).all())
    for t in counts:
        assert torch.equal(run(t), want), t
    # one row's own numbers are none: the rows beside it keep their bits
    bad = min(1, share - 1)
    store[table[bad, pp:].long()] = float("inf")
    store[table[bad, pp].long(), 0, ::3] = float("nan")
    want = run(1)
    others = torch.arange(R, device="cuda") != bad
    assert bool(torch.isfinite(want[others]).all())
    for t in counts:
        assert torch.equal(run(t)[others], want[others]), t
