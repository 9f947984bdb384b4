"""Requests of one StepRunner stepped from threads of their own, each on its own stream, against the general path, bit for bit."""

import threading

import pytest
import torch

from test_gpu_step_graph import _model, _plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,dtype", [("gpt", torch.float32), ("gpt", torch.bfloat16), ("kipolix", torch.bfloat16)])
def test_requests_from_their_own_threads(family, dtype):
    """Three threads: the first steps of one (launches, then a recording) fall among the others' launches and replays."""
    from diff_gpt_b200 import StepRunner

    model, V = _model(family, dtype)
    ids = {k: torch.randint(0, V, (48,), generator=torch.Generator().manual_seed(k)).tolist() for k in range(3)}
    want = {}
    for k, t in ids.items():
        cache = model.new_cache()
        cache.reset()
        with torch.inference_mode():
            want[k] = torch.cat([_plain(model, cache, t[:6])] + [_plain(model, cache, [x]) for x in t[6:]])
    runner, got, errors, go = StepRunner(model), {k: [] for k in ids}, [], threading.Barrier(len(ids))

    def follow(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                go.wait(20)
                got[k].append(runner.step(k, ids[k][:6], [5]))
                for x in ids[k][6:]:
                    got[k].append(runner.step(k, [x], [0]))
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=follow, args=(k,)) for k in ids]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(one.graph is not None for one in runner._single.values())
    for k in ids:
        assert torch.equal(torch.cat(got[k]), want[k]), k
