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


def test_one_request_on_two_streams():
    """A small fp32 GPT, whose tokens are replayed on the caller's stream: the streams take turns without synchronising, past the 256 and 512 keys
    where another plan takes over, around portions and where the cache grows; a second request takes the cache over."""
    from diff_gpt_b200 import GPT, StepRunner

    torch.manual_seed(0)
    model = GPT(vocab_size=128, n_embd=64, block_size=2048, n_head=4, n_layer=2)
    for p in model.parameters():
        torch.nn.init.normal_(p, std=0.1)
    model = model.cuda().eval()
    streams, runner = [torch.cuda.Stream() for _ in range(2)], StepRunner(model)
    for seed in range(2):
        ids = torch.randint(0, 128, (530,), generator=torch.Generator().manual_seed(seed)).tolist()
        portions, at, got, ends = {0: 200, 240: 3, 300: 180}, 0, [], []
        torch.cuda.synchronize()
        while at < len(ids):
            n = portions.get(at, 1)
            with torch.cuda.stream(streams[len(ends) % 2]):
                if len(ends) % 7 == 0:
                    torch.cuda._sleep(4_000_000)  # 2 ms in which the other stream would run ahead
                got.append(runner.step("r", ids[at : at + n], [n - 1]))
            at += n
            ends.append(at - 1)
        torch.cuda.synchronize()
        runner.finish("r")
        with torch.inference_mode():
            want = model(torch.tensor([ids], device="cuda"))[0][0, ends]
        assert all(one.graph is not None for one in runner._single.values())
        err = (torch.cat(got) - want).norm(dim=1) / want.norm(dim=1)
        assert bool((err < 1e-5).all()), err.max()  # fp32, sums in another order
