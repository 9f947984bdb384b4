"""Every tile form of dgpt_linear (single CTAs of 64, 128, 192 and 256 columns, CTA pairs of 128, 192 and 256) with every storing epilogue,
at sizes that end inside a tile in each direction."""

import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K) and the form that gemm_run takes for them on 148 multiprocessors: columns of a tile, CTAs of one
FORMS = {
    "one CTA, 64": ((100, 272, 136), (64, 1)), "one CTA, 64, two rows of tiles": ((300, 272, 200), (64, 1)),
    "one CTA, 128": ((33, 9584, 72), (128, 1)), "one CTA, 192": ((1990, 1584, 72), (192, 1)), "one CTA, 256": ((1990, 2256, 72), (256, 1)),
    "one CTA, 256, several rounds": ((4500, 2320, 328), (256, 1)), "pair, 128": ((555, 2064, 2056), (128, 2)),
    "pair, 192": ((1100, 2064, 2056), (192, 2)), "pair, 256": ((1100, 3088, 1032), (256, 2)), "pair, several rounds": ((4500, 2320, 1032), (256, 2)),
    "one row": ((1, 16, 8), None), "one row, shared K": ((1, 528, 1032), None), "one row, a warp a pair": ((1, 4752, 264), None),
    "two rows, shared K": ((2, 1008, 5456), None), "two rows, a warp a pair": ((2, 4752, 520), None), "three rows": ((3, 48, 24), (64, 1)),
}


def _form(M, N, K):
    """gemm_run's rule, restated: the least of rounds x clocks of a tile, 4000 more for a pair."""
    best = []
    for bn, cg in ((256, 2), (192, 2), (128, 2), (256, 1), (192, 1), (128, 1), (64, 1)):
        if cg == 1 or M > 128:
            tiles = -(-M // (128 * cg)) * -(-N // bn)
            block = max(2 * bn, (16384 + bn // cg * 128) / 56)
            best.append((-(-tiles // (148 // cg)) * max(-(-K // 64) * block, 16 * bn) + 4000 * (cg - 1), (bn, cg)))
    return min(best, key=lambda x: x[0])[1]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("epilogue", ["plain", "swiglu", "add", "xielu", "silu_gate", "softcap"])
def test_every_form_and_epilogue(form, epilogue):
    """Rounded once from fp32 sums (plain, add, xielu, silu_gate): half a bf16 step (8 significant bits: 2^-8 of the value), and 2^-20 of the sum's terms for
    the fp32 order.  swiglu rounds to bf16 inside: bit for bit the library's own
    element-wise kernel on the plain output.  softcap: three roundings to bf16 of the quotient, the tangent and the product, and 2^-21
    absolute in the tangent (its exponential form)."""
    from diff_gpt_b200 import ops

    (M, N, K), taken = FORMS[form]
    assert taken is None or _form(M, N, K) == taken
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * 0.3).bfloat16()
    r = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    half = epilogue in ("swiglu", "silu_gate")
    wide = torch.full((M + 1, (N // 2 if half else N) + 64), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = wide[:M, 32 : 32 + (N // 2 if half else N)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = {"plain": {}, "swiglu": dict(swiglu=(1.702, 7.0)), "add": dict(add=r), "xielu": dict(xielu=(0.8, 1.2)),
          "silu_gate": dict(silu_gate=True), "softcap": dict(softcap=15.0)}[epilogue]
    ops.linear(a, w, out, status=status, **kw)
    assert status.item() == 0
    assert torch.isnan(wide[M:].float()).all() and torch.isnan(wide[:, :32].float()).all() and torch.isnan(wide[:, 32 + out.shape[1] :].float()).all()
    if epilogue in ("swiglu", "softcap"):
        plain = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        ops.linear(a, w, plain)
        if epilogue == "softcap":
            want = 15.0 * torch.tanh(plain.double() / 15.0)
            assert bool(((out.double() - want).abs() <= 3 * 2.0**-8 * 1.01 * want.abs() + 15 * 2.0**-21).all())
        else:
            want = torch.empty((M, N // 2), dtype=torch.bfloat16, device="cuda")
            ops.swiglu(plain, want, 1.702, 7.0)
            assert torch.equal(out, want)
        return
    z = a.double() @ w.double().T
    terms = a.double().abs() @ w.double().abs().T
    if epilogue == "add":
        want = z + r.double()
    elif epilogue == "xielu":
        want = torch.where(z > 0, 0.8 * z * z, 1.2 * (torch.expm1(z.clamp(max=0)) - z.clamp(max=0))) + z / 2
        terms = terms * (1 + 1.6 * z.abs())  # slope of the curve
    elif epilogue == "silu_gate":
        gate, up = z[:, 0::2], z[:, 1::2]
        want = torch.nn.functional.silu(gate) * up
        terms = 1.1 * terms[:, 0::2] * up.abs() + gate.abs() * terms[:, 1::2]
    else:
        want = z
    bound = want.abs() * (2.0**-8 + 2.0**-18) + terms * 2.0**-20 + 2.0**-30
    assert bool(((out.double() - want).abs() <= bound).all()), ((out.double() - want).abs() / bound).max().item()
