"""When a configured model's packed weights are made anew."""

import pytest
import torch

import delunex_cases
import kipolix_cases


@pytest.mark.parametrize("cases", [delunex_cases, kipolix_cases])
def test_parametrized_weight_is_packed_again_after_a_change(cases):
    """A weight behind a parametrization is no parameter of the model itself any more; its original, below it, still counts."""
    model = cases.build(cases.CASES["tiny"], 3, torch.float32, device="cpu")[0]
    name = next(n for n, _ in model.named_parameters() if n.endswith("mix__o"))

    class Twice(torch.nn.Module):
        def forward(self, w):
            return 2 * w

    torch.nn.utils.parametrize.register_parametrization(model, name, Twice())
    first = model.packed_weights()
    assert model.packed_weights() is first
    with torch.no_grad():
        model.parametrizations[name].original.add_(1.0)
    second = model.packed_weights()
    assert second is not first and not torch.equal(second.layers[0].w_o_t, first.layers[0].w_o_t)


@pytest.mark.parametrize("cases", [delunex_cases, kipolix_cases])
def test_a_parameter_set_to_none_is_passed_over(cases):
    model = cases.build(cases.CASES["tiny"], 3, torch.float32, device="cpu")[0]
    model.register_parameter("extra", None)
    assert model.packed_weights() is model.packed_weights()
