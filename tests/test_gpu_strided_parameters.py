"""Layer weights that are column slices of a wider buffer, or transposed, give what contiguous ones give, up to the order of the sums."""

import pytest
import torch

from test_gpu_step_graph import _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,dtype", [("gpt", torch.float32), ("gpt", torch.bfloat16), ("delunex", torch.bfloat16), ("kipolix", torch.bfloat16)])
@pytest.mark.parametrize("how", ["odd row stride", "transposed"])
def test_short_prompts_and_single_tokens(family, dtype, how):
    """A prompt of 11 tokens and single tokens behind it (launches, then a recording).  bf16: another order of the sums in three
    layers moved a logit by 4 % of the largest where cuBLAS took every product; twice that is allowed."""
    from diff_gpt_b200 import StepRunner

    model, V = _model(family, dtype)
    ids = torch.randint(0, V, (14,), generator=torch.Generator().manual_seed(3)).tolist()

    def run():
        runner = StepRunner(model)
        return torch.cat([runner.step("r", ids[:11], [10])] + [runner.step("r", [t], [0]) for t in ids[11:]])

    want = run()
    table = model.token_embedding_table.weight if family == "gpt" else None
    for name, p in model.named_parameters():
        if p.dim() == 2 and p.shape[0] > 1 and p is not table and name not in ("embed", "head", "bigram"):
            if how == "transposed":
                p.data = p.data.t().contiguous().t()
            else:
                wide = torch.empty(p.shape[0], p.shape[1] + 1, dtype=dtype, device="cuda")
                wide[:, :-1].copy_(p.detach())
                p.data = wide[:, :-1]
    got = run()
    assert (got - want).abs().max().item() <= (1e-5 if dtype == torch.float32 else 8e-2) * want.abs().max().item()
