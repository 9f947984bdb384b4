"""fp32 linear layers and warp-level attention of small models: dgpt_linear_f32 at the edges of its tiles, and attention whose queries
are shared by eight lanes, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 2, 4), (16, 32, 64), (17, 34, 68), (100, 256, 64), (15, 62, 128), (33, 30, 132), (100, 64, 300), (5, 512, 512)])
@pytest.mark.parametrize("epilogue", ["plain", "swiglu", "add", "softcap"])
def test_linear_f32(M, N, K, epilogue):
    """Sums of K terms in fp32: 2^-22 of the terms' size (a chain of K / 16 and three more additions), carried through the epilogue."""
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    wide_a = torch.randn(M, K + 8, generator=g, device="cuda")
    a, w, r = wide_a[:, 4 : 4 + K], torch.randn(N, K, generator=g, device="cuda"), torch.randn(M, N, generator=g, device="cuda")
    half = epilogue == "swiglu"
    wide = torch.full((M + 1, (N // 2 if half else N) + 3), float("nan"), device="cuda")
    out = wide[:M, 1 : 1 + (N // 2 if half else N)]
    z, terms = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    if epilogue == "add":
        out.copy_(r)  # in place
    ops.linear_f32(a, w, out, **{"plain": {}, "swiglu": dict(swiglu=(1.702, 7.0)), "add": dict(add=out), "softcap": dict(softcap=15.0)}[epilogue])
    if epilogue == "add":
        z = z + r.double()
    elif epilogue == "softcap":
        z = 15 * torch.tanh(z / 15)
    elif half:
        gate, lin = z[:, 0::2].clamp(max=7), z[:, 1::2].clamp(-7, 7)
        z = gate * torch.sigmoid(1.702 * gate) * (lin + 1)
        terms = 1.2 * terms[:, 0::2] * 8 + gate.abs() * terms[:, 1::2]
    assert torch.isnan(wide[M]).all() and torch.isnan(wide[:, 0]).all() and torch.isnan(wide[:, 1 + out.shape[1] :]).all()
    assert bool(((out.double() - z).abs() <= terms * 2.0**-20 + z.abs() * 2.0**-20 + 1e-6).all())


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.bfloat16, 8e-3)])
@pytest.mark.parametrize("D", [8, 16, 32])
@pytest.mark.parametrize("B,H,Tq,Tk,causal", [(1, 4, 100, 89, False), (2, 3, 17, 17, True), (1, 2, 1, 1, True), (1, 4, 16, 70, True), (3, 2, 33, 31, False)])
def test_shared_queries(B, H, Tq, Tk, causal, D, dtype, tol):
    """Rounded once from fp32 sums; the lanes' shares differ in size and some see no key at all."""
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(Tq + Tk + D)
    q = torch.randn(B, Tq, H, D, generator=g, device="cuda").to(dtype)
    kv = torch.randn(2, B, H, Tk, D, generator=g, device="cuda").to(dtype)
    y = torch.full((B, Tq, H, D), float("nan"), dtype=dtype, device="cuda")
    lse = torch.empty(B * Tq, H, device="cuda")
    lay = ops.kv_layout(kv[0], kv[1], H * Tk * D, Tk * D, Tk)
    C, off = H * D, Tk - Tq if causal else 0
    ops.fmha_prefill(q, lay, y, B=B, H=H, Tq=Tq, D=D, q_batch_stride=Tq * C, q_row_stride=C, o_batch_stride=Tq * C, o_row_stride=C,
                     kv_len_all=Tk, q_offset=off, causal=causal, lse=lse, impl=1)
    s = torch.einsum("bqhd,bhkd->bhqk", q.double(), kv[0].double()) * D**-0.5
    if causal:
        s = s.masked_fill(torch.arange(Tk, device="cuda") > torch.arange(Tq, device="cuda")[:, None] + off, float("-inf"))
    want = torch.einsum("bhqk,bhkd->bqhd", torch.softmax(s, -1), kv[1].double())
    assert (y.double() - want).abs().max().item() <= tol * max(1.0, want.abs().max().item())
    assert (lse.view(B, Tq, H).transpose(1, 2).double() - torch.logsumexp(s, -1)).abs().max().item() <= 1e-5
