"""What a user puts on the way of a GPT's forward sees single tokens of a StepRunner too, also after some were recorded."""

import pytest
import torch

from test_gpu_step_graph import _model

pytestmark = pytest.mark.gpu


def test_hook_and_replaced_forward_see_every_token():
    from diff_gpt_b200 import StepRunner

    model, _ = _model("gpt", torch.float32)
    runner, seen = StepRunner(model), []
    runner.step("r", [1, 2, 3], [2])
    for t in range(4):
        runner.step("r", [t], [0])
    hook = model.register_forward_hook(lambda m, args, out: (out[0] * 2, out[1]))
    doubled = runner.step("r", [5], [0])
    hook.remove()
    plain = StepRunner(model)
    for tokens in ([1, 2, 3], [0], [1], [2], [3]):
        plain.step("r", tokens, [len(tokens) - 1])
    assert torch.equal(doubled, 2 * plain.step("r", [5], [0]))
    inner = model.forward
    model.forward = lambda *a, **k: (seen.append(1), inner(*a, **k))[1]
    for t in range(3):
        runner.step("r", [t], [0])
    assert len(seen) == 3
