"""The numbers that a GPT carries beside its weights are read again by every token of a StepRunner."""

import pytest
import torch

from test_gpu_step_graph import _model, _plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name,value", [("logit_softcap", 2.0), ("logit_softcap", 0.0), ("swiglu_alpha", 0.3), ("swiglu_limit", 0.05)])
def test_changed_between_recorded_tokens(name, value, dtype):
    from diff_gpt_b200 import StepRunner

    model, _ = _model("gpt", dtype)
    runner, cache = StepRunner(model), model.new_cache()
    cache.reset()
    with torch.inference_mode():
        for at, tokens in enumerate([[1, 2, 3]] + [[t] for t in range(10)]):
            if at == 6:
                setattr(model, name, value)
            got = runner.step("r", tokens, [len(tokens) - 1])
            assert torch.equal(got, _plain(model, cache, tokens)), at
