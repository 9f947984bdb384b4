"""StepRunner's host logic without a GPU: streams, graphs and the model are stand-ins that note who is inside."""

import contextlib
import gc
import threading
import time
import weakref
from types import SimpleNamespace

import pytest
import torch


class _Logits:
    def to(self, *a, **k):
        return SimpleNamespace(record_stream=lambda s: None)


class _Storage:
    """Stands for a cache's tensor, or for packed weights."""


class _Busy:
    """What is enqueued on the runner's stream: only one thread may be at it."""

    def __init__(self):
        self.inside, self.overlaps = set(), 0

    def work(self):
        me = threading.get_ident()
        self.overlaps += bool(self.inside - {me})
        self.inside.add(me)
        time.sleep(0.002)
        self.inside.discard(me)


@pytest.fixture
def cuda(monkeypatch):
    class Graph:
        def capture_begin(self, **k):
            pass

        def capture_end(self):
            pass

        def replay(self):
            pass

    stream = SimpleNamespace(wait_stream=lambda other: None, synchronize=lambda: None)
    monkeypatch.setattr(torch.cuda, "Stream", lambda **k: stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: stream)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)


def _model(busy):
    from diff_gpt_b200.model.gpt import SingleStep

    class Cache:
        def __init__(self):
            self.storage = _Storage()

        def reset(self):
            self.pos = 0

    class Plan:
        logits = _Logits()

        def run(self, ids, bind):
            busy.work()

    class Model:
        vocab_size, embedding = 8, torch.zeros(1)

        def __init__(self):
            self.last_packed = _Storage()

        def new_cache(self):
            return Cache()

        def single_step_allowed(self):
            return True

        def cache_storage(self, cache):
            return (cache.storage,)

        def single_step(self, cache, old, stream):
            held = (self.last_packed, cache.storage)
            if old is not None and old.fits((0,), held):
                return old
            return SingleStep(Plan(), None, torch.zeros(4, dtype=torch.int32), (0,), held, checks=False)

        def logits_at(self, idx, cache, rows):
            cache.pos += idx.shape[1]
            return torch.zeros(rows.numel(), 8)

    return Model()


def _in_thread(fn):
    err = []

    def go():
        try:
            fn()
        except Exception as e:  # noqa: BLE001
            err.append(e)

    t = threading.Thread(target=go)
    t.start()
    return t, err


def test_one_thread_at_a_time_on_the_runners_stream(cuda):
    from diff_gpt_b200 import StepRunner

    busy = _Busy()
    runner = StepRunner(_model(busy))
    threads = [_in_thread(lambda r=r: [runner.step(r, [1], [0]) for _ in range(8)]) for r in range(4)]
    for t, err in threads:
        t.join()
        assert not err
    assert busy.overlaps == 0
    assert sorted(c.pos for c in runner._live.values()) == [8] * 4


def test_a_thread_records_only_after_a_step_of_its_own(cuda):
    """Thread B takes over a request that A has begun: B's first step runs as launches, its second is recorded."""
    from diff_gpt_b200 import StepRunner

    runner = StepRunner(_model(_Busy()))
    runner.step("r", [1], [0])
    seen = []

    def b():
        for _ in range(2):
            runner.step("r", [1], [0])
            seen.append(next(iter(runner._single.values())).graph is not None)

    t, err = _in_thread(b)
    t.join()
    assert not err and seen == [False, True]


def test_replaced_methods_and_hooks_keep_the_general_path():
    import delunex_cases
    from diff_gpt_b200 import GPT
    from diff_gpt_b200.model.registry import model_class

    kw = dict(vocab_size=64, n_embd=32, n_head=2, n_layer=1)
    cfg = delunex_cases.CASES["tiny"]
    other = model_class(cfg)
    assert GPT(**kw).single_step_allowed() and other.from_config(cfg).single_step_allowed()

    class Own(GPT):
        def forward(self, *a, **k):
            return super().forward(*a, **k)

    class OwnOther(other):
        def logits_at(self, *a):
            return super().logits_at(*a)

    assert not Own(**kw).single_step_allowed() and not OwnOther.from_config(cfg).single_step_allowed()
    m = GPT(**kw)
    m.forward = lambda *a, **k: None
    assert not m.single_step_allowed()
    for add in (m.register_forward_hook, m.register_forward_pre_hook, torch.nn.modules.module.register_module_forward_hook):
        m = GPT(**kw)
        h = (getattr(m, add.__name__) if hasattr(m, add.__name__) else add)(lambda *a: None)
        assert not m.single_step_allowed()
        h.remove()
        assert m.single_step_allowed()
    # the module itself is not called on the way to the other models' logits
    m = other.from_config(cfg)
    m.register_forward_hook(lambda *a: None)
    assert m.single_step_allowed()


@pytest.mark.parametrize("tokens", [[1], [1, 2, 3]])
def test_replaced_weights_and_outgrown_storage_are_let_go(cuda, tokens):
    """By the next step, a single token or a portion: the storage of that request's cache, and the weights that every recording held."""
    from diff_gpt_b200 import StepRunner

    model = _model(_Busy())
    runner = StepRunner(model)
    for r in ("a", "b"):
        for _ in range(3):
            runner.step(r, [1], [0])
    cache = runner._live["a"]
    storage, weights = weakref.ref(cache.storage), weakref.ref(model.last_packed)
    cache.storage, model.last_packed = _Storage(), _Storage()
    runner.step("a", tokens, [0])
    gc.collect()
    assert storage() is None and weights() is None
    assert all(one.held[0] is model.last_packed for one in runner._single.values())


class _Line:
    """A stream that knows which pieces of work it, and what it has waited for, have behind them."""

    def __init__(self, number):
        self.cuda_stream, self.behind = number, set()

    def wait_stream(self, other):
        self.behind |= other.behind

    def __ne__(self, other):  # as torch's streams, whose `!=` may be False where `==` is False too
        return False

    def synchronize(self):
        pass


@pytest.mark.parametrize("whole", [True, False])
def test_a_request_that_moves_from_stream_to_stream(monkeypatch, whole):
    """Every step runs behind the one before, also where the plan changes (every fifth token), where the cache grows and around portions."""
    from diff_gpt_b200 import StepRunner, ops
    from diff_gpt_b200.model.gpt import SingleStep

    callers, current, recording = [_Line(1), _Line(2)], [None], [False]
    done, missed = [0], []

    def work():
        if not recording[0]:
            line = current[0]
            missed.extend(set(range(done[0])) - line.behind)
            line.behind.add(done[0])
            done[0] += 1

    class Graph:
        def capture_begin(self, **k):
            recording[0] = True

        def capture_end(self):
            recording[0] = False

        def replay(self):
            work()

    @contextlib.contextmanager
    def on(line):
        was, current[0] = current[0], line
        yield
        current[0] = was

    monkeypatch.setattr(torch.cuda, "Stream", lambda **k: _Line(9))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: current[0])
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)
    monkeypatch.setattr(ops, "_stream", lambda: current[0].cuda_stream)

    class Cache:
        def reset(self):
            self.pos = 0

    class Tensor(_Logits):
        def copy_(self, x):
            pass

        def record_stream(self, s):
            pass

    class Model:
        vocab_size, embedding, last_packed = 8, torch.zeros(1), _Storage()
        new_cache = Cache
        single_step_allowed = lambda self: True  # noqa: E731
        cache_storage = lambda self, cache: ()  # noqa: E731

        def single_step(self, cache, old, stream):
            kind = (cache.pos // 5,)
            if old is not None and old.fits(kind, (self.last_packed,)):
                return old
            work()  # the storage grows
            plan = SimpleNamespace(whole=whole, logits=Tensor(), status=Tensor(), run=lambda ids, bind: work())
            return SingleStep(plan, SimpleNamespace(len0=Tensor()), Tensor(), kind, (self.last_packed,), checks=False)

        def logits_at(self, idx, cache, rows):
            work()
            cache.pos += idx.shape[1]
            return torch.zeros(rows.numel(), 8)

    monkeypatch.setattr(SingleStep, "enqueue", lambda self: self.plan.run(None, None))
    runner = StepRunner(Model())
    for request in ("a", "b"):  # b takes a's cache over
        for i, n in enumerate([3, 1, 1, 1, 1, 1, 1, 1, 1, 2, 1, 1, 1, 1, 4, 1, 1, 1]):
            with on(callers[i // 2 % 2 if i < 9 else i % 2]):
                runner.step(request, [1] * n, [0])
        runner.finish(request)
    assert done[0] > 36 and not missed, missed
