"""Linear layers of every tile form launched one behind the other, many times: a CTA that left before all that its pair's other half sends it
had arrived would disturb the one that takes its place."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [1, 2])
def test_results_do_not_depend_on_the_neighbours(streams):
    from diff_gpt_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(1)
    shapes = [(1100, 3088, 1032), (300, 272, 72), (1100, 2064, 2056), (129, 528, 8), (555, 2064, 2056), (4500, 2320, 1032), (1990, 2256, 72)]
    work = []
    for M, N, K in shapes:
        a, w = (torch.randn(r, K, generator=g, device="cuda").bfloat16() for r in (M, N))
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        ops.linear(a, w, out)
        work.append((a, w, out, out.clone()))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    lanes = [torch.cuda.Stream() for _ in range(streams)]
    for i in range(60):
        for k, (a, w, out, _) in enumerate(work):
            with torch.cuda.stream(lanes[k % streams]):
                out.fill_(float("nan"))
                ops.linear(a, w, out, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0
    for _, _, out, want in work:
        assert torch.equal(out, want)
