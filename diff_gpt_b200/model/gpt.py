"""Drop-in `GPT` whose inference forward runs on the libdgpt_b200 kernels.

Same constructor keywords, attributes and state_dict keys as the reference
module (src/diff_gpt/model/gpt.py:79-136), so checkpoints move both ways, and
the same `forward(idx, targets=None, kv_cache=None) -> (logits, loss)` contract
that the reference Engine and DiffGPT facade rely on (gpt.py:140-200).

The sub-modules below are parameter containers: they give the parameters their
reference names and shapes; the arithmetic of a forward pass is enqueued by
`ForwardPlan.run`, which walks the layers and launches

    embed+rmsnorm -> [depth-mix+rmsnorm -> QKVG GEMM -> rope/qk-norm/kv-append ->
    attention (+gate) -> out-proj GEMM -> depth-mix+rmsnorm -> FFN GEMM -> swiglu ->
    FFN GEMM (+residual)] x L -> rmsnorm -> tied-embedding GEMM -> soft-cap

Large bf16 products without an epilogue, and large fp32 ones, are on cuBLAS (torch.mm / addmm_).  The bf16 head and feed-forward
up projection, products of one bf16 row, those of small fp32 models (`own_f32`) and everything else are this library's.
There is no CPU implementation: CPU tensors raise.
"""

from __future__ import annotations

from abc import ABC, abstractmethod
from dataclasses import dataclass, field

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.nn.modules.module import _has_any_global_hook

from .. import ops
from .._lib import region
from ..sampler.sampler import Sampler
from .kv_cache import KVCache, PagedKVCache
from .rope import precompute_freqs_cis


class BaseGPT(nn.Module, ABC):
    """The seam the Engine and the DiffGPT facade program against (gpt.py:38-76)."""

    def __init__(self, block_size: int, vocab_size: int, n_embd: int, n_head: int, n_layer: int) -> None:
        super().__init__()
        self.block_size = block_size
        self.vocab_size = vocab_size
        self.n_embd = n_embd
        self.n_head = n_head
        self.n_layer = n_layer

    @abstractmethod
    def forward(self, idx, targets=None, kv_cache=None):
        ...

    @abstractmethod
    def generate(self, idx, max_new_tokens, sampler, seed=None):
        ...

    @property
    @abstractmethod
    def device_type(self) -> str:
        ...


class LateStatus:
    """A status word in pinned host memory for launches that nobody waits for: a kernel writes there only when something went wrong, and the
    host looks without a copy or a wait, when it next comes by.  Copies and pickles of its owner get one of their own."""

    def __init__(self) -> None:
        self._word = self._view = None

    def word(self) -> torch.Tensor | None:
        """The word, or None where it cannot be made now (a stream is being captured)."""
        if self._word is None and not torch.cuda.is_current_stream_capturing():
            self._word = torch.zeros(1, dtype=torch.int32).pin_memory()
            self._view = self._word.numpy()
        return self._word

    @property
    def used(self) -> bool:
        return self._word is not None

    def check(self) -> None:
        if self._view is not None and self._view[0]:
            bad, self._view[0] = int(self._view[0]), 0
            raise RuntimeError(f"device-side status {bad}: in an earlier forward a cache slot or position was out of range, or a bounded wait ran out; "
                               "its logits are not to be used")

    def __deepcopy__(self, memo) -> "LateStatus":
        return LateStatus()

    def __reduce__(self):
        return LateStatus, ()


class DeviceModel(BaseGPT):
    """A model whose forward is enqueued by a plan of this library's kernels: what the Engine, the step-by-step
    runner and the facade need from it, whatever its layers are."""

    logit_softcap: float = 0.0

    @property
    @abstractmethod
    def embedding(self) -> torch.Tensor:
        """The token table [V, C]; its device and dtype are the model's."""

    @abstractmethod
    def packed_weights(self):
        """Weights as the kernels want them, `head` [V, C] (the output head; the token table where they are tied) among
        them; the same object until a parameter is modified or moved."""

    @property
    def last_packed(self):
        """What `packed_weights` gave last, without a look at the parameters."""
        return self._packed

    # -- requests fed step by step --
    @abstractmethod
    def new_cache(self, batch_size: int = 1, seq_len: int = 0):
        """An empty cache with `reset()` and `get_pos()` for `forward(idx, kv_cache=...)`."""

    @abstractmethod
    def logits_at(self, idx: torch.Tensor, cache, rows: torch.Tensor) -> torch.Tensor:
        """Run idx (1, T) behind what `cache` holds; the logits [len(rows), V] of the given places among the T tokens."""

    # (class, method) that `logits_at` goes through up to the launches, itself first
    step_path: tuple = ()

    def single_step_allowed(self) -> bool:
        """Whether a token through `logits_at` is this library's launches and nothing else: none of the methods on the way
        replaced by a subclass or on the object and, where the module is called, no hook on it."""
        for cls, name in self.step_path:
            if name == "__call__":
                if self._forward_hooks or self._forward_pre_hooks or self._compiled_call_impl or _has_any_global_hook():
                    return False
            if getattr(type(self), name) is not getattr(cls, name) or name in self.__dict__:
                return False
        return bool(self.step_path)

    def cache_storage(self, cache) -> tuple:
        """The tensors of a cache from `new_cache` that are replaced when it grows."""
        return ()

    def single_step(self, cache, old: "SingleStep | None", stream: torch.cuda.Stream) -> "SingleStep | None":
        """The launches of one more token behind `cache`, which has room for it afterwards: `old` where it still fits, or None
        where a single token takes the general path.  What it allocates for itself belongs to `stream`, where it will run."""
        return None

    # what launches that nobody has waited for have to report, if the model has such
    late_status: LateStatus | None = None

    # -- batched decode (DecodeRun) --
    @abstractmethod
    def paged_cache(self, n_series: int, rows_per_series: int, prefix_len: int, max_new: int, page_tokens: int, pool=None):
        """The cache of a decode run: prompt pages shared by a series' rows, private pages per row."""

    @abstractmethod
    def prefill_plan(self, cache, members: list[int], P: int, fmha_impl: int, few_rows: bool = True):
        """(binding, plan) that prefills the P-token prompts of the series `members` into `cache`.  `few_rows`: one or two rows may
        run on kernels of their own, whose bf16 sums have another order than a larger batch's."""

    @abstractmethod
    def decode_plan(self, cache, prompt_lens: torch.Tensor, max_keys: int, step: torch.Tensor, shared: bool, fmha_impl: int,
                    overlap_prefix: bool, want_logits: bool, few_rows: bool = True):
        """(binding, plan) of one decode step of all rows; `step` is the device counter of generated tokens."""


# ---- parameter containers (names and shapes of the reference state_dict) -------
class SwiGLU(nn.Module):
    def __init__(self, alpha: float, limit: float) -> None:
        super().__init__()
        self.alpha = alpha
        self.limit = limit

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        out = torch.empty((*x.shape[:-1], x.shape[-1] // 2), dtype=x.dtype, device=x.device)
        ops.swiglu(x.contiguous(), out, self.alpha, self.limit)
        return out


class FeedForward(nn.Module):
    def __init__(self, n_embd: int, swiglu_alpha: float, swiglu_limit: float) -> None:
        super().__init__()
        self.net = nn.Sequential(
            nn.Linear(n_embd, 4 * n_embd, bias=False),
            SwiGLU(alpha=swiglu_alpha, limit=swiglu_limit),
            nn.Linear(2 * n_embd, n_embd, bias=False),
        )


class MultiHeadAttention(nn.Module):
    def __init__(self, n_embd: int, n_head: int, layer_idx: int) -> None:
        super().__init__()
        assert n_embd % n_head == 0
        assert (n_embd // n_head) % 2 == 0  # RoPE rotates pairs
        self.n_embd, self.n_head, self.layer_idx = n_embd, n_head, layer_idx
        self.head_dim = n_embd // n_head
        for name in ("c_q", "c_k", "c_v", "c_g", "c_proj"):
            setattr(self, name, nn.Linear(n_embd, n_embd, bias=False))


class Block(nn.Module):
    def __init__(self, n_embd, n_head, swiglu_alpha, swiglu_limit, layer_idx, layers_per_block=1) -> None:
        super().__init__()
        assert layers_per_block >= 1
        self.layer_idx = layer_idx
        self.layers_per_block = layers_per_block
        self.sa = MultiHeadAttention(n_embd=n_embd, n_head=n_head, layer_idx=layer_idx)
        self.ffwd = FeedForward(n_embd=n_embd, swiglu_alpha=swiglu_alpha, swiglu_limit=swiglu_limit)
        self.attn_res_proj = nn.Linear(n_embd, 1, bias=False)
        self.mlp_res_proj = nn.Linear(n_embd, 1, bias=False)


CACHE_NORMS = True  # depth mix: reuse the norm factors of committed candidates instead of recomputing them
FUSED_FFN = True  # first feed-forward GEMM on the library's tcgen05 kernel with the SwiGLU fused (bf16 only)
FUSED_FFN_MIN_ROWS = 256
# The shared-prompt attention phase while it runs beside the per-row phase: which kernel (an `impl` of
# dgpt_fmha_prefill) and on how many SMs.  Measured per 255 config-4 steps, one process, alternating: the persistent
# kernel with two query tiles per CTA on 64 SMs, which it owns outright (it fills an SM's shared memory and TMEM)
# while the HBM-bound per-row kernel has the other 84 to itself, 1249-1259 ms; on 48 or 80 SMs 1256-1262; the small
# kernel (impl 3) on every SM, one CTA each, sharing the SMs with the per-row kernel, 1271-1275; the persistent kernel
# with one query tile per CTA on 64 SMs 1267-1271, on 40 SMs 1288 (the phase becomes the longer one).  Where the prompt
# phase is the longer one it takes more SMs: see `prefix_ctas`.
PREFIX_CTAS = 64
PREFIX_IMPL = 4


def prefix_ctas(units: int, key_tiles: int, own_us: float, n_sm: int) -> int:
    """SMs for the shared-prompt phase: `units` work items (pairs of 128-query tiles) of `key_tiles` 128-key tiles, about 3.3 us a
    tile, beside a per-row phase that takes `own_us` on the whole GPU and meanwhile advances on the SMs left over.  PREFIX_CTAS,
    unless one SM per unit, or every SM, is estimated to be done earlier.  Measured per layer with the merge, us: 3 x 333 rows,
    12 heads, 777 + 20 keys (72 units) on 64 SMs 42.5, on 72 34.1; 10 x 64 rows, 8 heads, 500 + 30 keys (80 units) 26.9 -> 19.0; 40 x
    20 rows, 12 heads, 1000 + 40 keys (480 units) 148, on all 92; 4096 rows, 12 heads, 1024 + 128 keys (192 units) 282, on all 295.  The rate a
    tile is that of heads of 64; with heads of 32 no step of twelve such jobs got slower (4 layers, us: 40 x 20 rows 505 -> 393, 20 x 33
    rows, 1400 keys 438 -> 360, 10 x 64 217 -> 176, 4096 rows 405 -> 400)."""

    def estimate(ctas: int) -> float:
        phase = -(-units // ctas) * key_tiles * 3.3
        return phase + max(0.0, own_us - phase * min(1.0, 1.3 * (n_sm - ctas) / n_sm))

    few = min(PREFIX_CTAS, n_sm)
    many = min(units, n_sm)
    return many if units > few and estimate(many) < 0.97 * estimate(few) else few


SIDE_PRIORITY = -1  # stream of the shared-prompt attention phase: ahead of the per-row phase it runs beside


@dataclass
class SingleStep:
    """One token of one request: a plan and a binding whose changing numbers are read from `numbers` on the device (token, slot,
    position, keys), so that the launches can be recorded once and replayed.

    kind    host-side choices and numbers that the launches were made with (key splits, soft-cap, ...)
    held    what the launches point at, the packed weights first; kept alive here and compared by `is`
    """

    plan: object
    bind: object
    numbers: torch.Tensor  # int32 [4]
    kind: tuple
    held: tuple
    checks: bool  # the plan's status is read after every step
    graph: torch.cuda.CUDAGraph | None = None
    launches: int = 0
    runs: int = 0
    streams: set = field(default_factory=set)  # handles of the streams that it was replayed on, but for the runner's

    def fits(self, kind: tuple, held: tuple) -> bool:
        return self.kind == kind and len(self.held) == len(held) and all(a is b for a, b in zip(self.held, held))

    def current(self, weights, storage: tuple) -> bool:
        """Whether it still holds these weights, and this storage of its cache."""
        return self.held[0] is weights and all(any(t is h for h in self.held) for t in storage)

    def enqueue(self) -> None:
        self.plan.run(self.numbers[0:1], self.bind)


def own_f32(M: int, N: int, K: int, ends: bool = False) -> bool:
    """Whether an fp32 product runs on dgpt_linear_f32; `ends`: it ends in an addition, a SwiGLU or a soft-cap, which cuBLAS leaves to
    a pass of its own (or a slower kernel).  Measured over C = 64 to 512 (K = C or 2 C, N = C to 4 C), us, cuBLAS / own:
    more than 16 rows, up to 400 tiles: 100 x 256 x 64 3.63 / 2.62, 100 x 64 x 128 4.65 / 2.93, 400 x 512 x 64 3.95 / 3.93, none over 3 % behind;
    beyond 1000 x 256 x 64 3.99 / 4.69, 400 x 1024 x 256 9.4 / 13.2.
    Up to 16 rows cuBLAS has kernels for few rows: 2 x 512 x 512 3.67 / 6.66, 8 x 256 x 256 3.29 / 4.16, 2 x 64 x 64 2.04 / 2.34.  Own there:
    with an ending up to K = 128 (2 x 512 x 128 SwiGLU 3.57 / 3.48, 8 x 256 x 64 2.9 / 2.3), from 8 wide rows on (8 x 1024 x 256 6.43 / 4.25,
    8 x 2048 x 512 9.63 / 7.00), one row up to K = 64 (1 x 256 x 64 2.90 / 2.28; 1 x 64 x 128 1.97 / 2.81), and from 5 rows on up to K = 64, level
    by itself (8 x 256 x 64 2.41 / 2.48) and 1 to 3 % ahead in a whole forecast of 5 to 12 futures."""
    if -(-M // 16) * -(-N // 32) > 400 or K > 512:
        return False
    if M > 16:
        return True
    if M == 1:
        return K <= 64
    return (ends and K <= 128) or (M >= 5 and K <= 64) or (M >= 8 and N >= 1024 and K >= 256)


def whole_f32(C: int, H: int, L: int, V: int, n_seq: int, T: int, keys: int) -> bool:
    """Whether a forward of an fp32 model runs as one launch of dgpt_small_gpt: `T` tokens of each of `n_seq` sequences behind one another,
    or one token of `n_seq` rows (T = 1), none of which sees more than `keys` keys.
    Decode steps, us a step, one launch per product / one for all: 2 layers of 64, 148 rows, 60 keys 69 / 14, 1900 keys 167 / 38; up to two
    rows a multiprocessor ahead at every number of keys (4 layers of 128, 296 rows, 1900 keys 406 / 260), up to four below a thousand
    (12 layers of 128, 592 rows, 900 keys 1193 / 1073, 1900 keys level), up to eight where the model is narrow (64, 1000 rows, 300 keys
    101 / 76, 900 keys 141 / 146; 128, 60 keys 211 / 189, 300 keys 246 / 295).  Every CTA reads all weights and its rows' prompt by itself.
    Whole sequences, us a call with its host work: 2 layers of 64, 1 x 256 tokens 520 / 256, 1 x 1024 590 / 979; 4 layers of 128, 1 x 128
    855 / 365, 1 x 512 983 / 1334; many sequences pay while their CTAs are two a multiprocessor (8 x 256 565 / 382, 32 x 64 578 / 247)."""
    if not ops.small_gpt_supported(C, H, L, V, keys):
        return False
    sms = _sm_count()
    if T == 1:
        return keys <= 2048 if n_seq <= 2 * sms else keys <= 1024 if n_seq <= 4 * sms else n_seq <= 8 * sms and C <= 64 and keys <= 512
    return T <= (256 if C <= 64 else 128) and keys <= 1024 and n_seq * -(-min(T, 128) // 8) <= 2 * sms


# ---- how one forward call is bound to K/V storage ----------------------------------
@dataclass
class KvBinding:
    """Where the new K/V go and which cached keys each query sees.

    layouts[l]    storage of layer l; its sequence index is the row of `pos0`
    pos0, slot0   int32 [n_seq]: RoPE position / cache slot of the first new token
    step          int32 device scalar added to both (None = 0)
    Prefill / chunk (T >= 1, `decode` False): keys [0, kv_len) with the causal rule j <= q_offset + i.
    Decode (T == 1, `decode` True): row r sees slots [0, len0[r]) and [start1[r], start1[r] + len1[r] + step).
    shared_*      optional shared-prefix phase: rows are grouped `rows_per_series` to a series whose
                  prompt keys live in `shared_layouts[l]` (sequence index = series), lengths `shared_len`.
    """

    layouts: list
    pos0: torch.Tensor
    slot0: torch.Tensor
    step: torch.Tensor | None = None
    decode: bool = False
    kv_len: int = 0
    q_offset: int = 0
    len0: torch.Tensor | None = None
    start1: torch.Tensor | None = None
    len1: torch.Tensor | None = None
    n_splits: int = 1
    shared_layouts: list | None = None
    shared_len: torch.Tensor | None = None
    shared_keys: int = 0  # the longest prompt, on the host
    own_keys: int = 0  # mean number of a row's own keys over the run, on the host
    rows_per_series: int = 0
    fmha_impl: int = 0
    overlap_prefix: bool = False  # run the shared-prompt phase on a second stream beside the per-row phase


class ForwardPlan:
    """Buffers for one (n_seq, T) forward and the launch sequence that fills them.

    `run` only enqueues work on the current stream and reuses the same buffers
    every time, so a plan can be captured into a CUDA graph and replayed.
    """

    def __init__(self, model: "GPT", n_seq: int, T: int, last_only: bool = False, want_logits: bool = True,
                 cap: float = 0.0, few_rows: bool = True, keys: int | None = None, late: bool = False) -> None:
        """`cap`: soft-cap the logits as they are stored (0 = raw logits).  `few_rows`: see `DeviceModel.prefill_plan`.  `keys`: the
        most keys that a token sees, where the kernel of small fp32 models may run the whole forward (see whole_f32).  `late`: nobody reads
        the plan's status; that kernel's goes to the model's `late_status`."""
        emb = model.token_embedding_table.weight
        dev, dt = emb.device, emb.dtype
        C, V, L = model.n_embd, model.vocab_size, model.n_layer
        n = n_seq * T
        self.model, self.n_seq, self.T, self.n, self.last_only = model, n_seq, T, n, last_only

        def buf(*shape, dtype=dt):
            return torch.empty(shape, dtype=dtype, device=dev)

        n_out = n_seq if last_only else n
        self.cap = cap
        self.logits = buf(n_out, V) if want_logits else None
        self.keys = keys
        self.whole = (
            keys is not None and want_logits and dt == torch.float32 and emb.is_contiguous() and whole_f32(C, model.n_head, L, V, n_seq, T, keys)
        )
        self.status = model.report() if late and self.whole else None
        if self.status is None:
            self.status = torch.zeros(1, dtype=torch.int32, device=dev)
        self.side = None
        if self.whole:
            return
        self.x, self.u, self.q, self.y = buf(n, C), buf(n, C), buf(n, C), buf(n, C)
        self.qkvg = buf(n, 4 * C)
        self.parts = [buf(n, C) for _ in range(L)]
        self.act = buf(n, 2 * C)
        self.xn = buf(n_out, C)
        self.last = buf(n_out, C) if (last_only and T > 1) else None
        # the tied-embedding head on the library's tcgen05 GEMM (bf16 with tileable sizes); fp32: see own_f32
        self.own_head = dt == torch.bfloat16 and C % 8 == 0 and V % 16 == 0
        # tcgen05 GEMM + SwiGLU epilogue: bf16 with tileable sizes, and enough rows to fill the tensor cores
        # parameters may be views: rows that the kernels for small products do not take stay on cuBLAS
        aligned = model.packed_weights().rows16
        self.few_rows = few_rows
        self.one_row = few_rows and dt == torch.bfloat16 and C % 16 == 0 and n == 1 and aligned  # see dgpt_linear: ahead of cuBLAS at every size
        self.fused_ffn = FUSED_FFN and dt == torch.bfloat16 and C % 8 == 0 and (n >= FUSED_FFN_MIN_ROWS or self.one_row)
        self.f32 = dt == torch.float32 and C % 4 == 0 and aligned
        self.own_ffn1 = self.f32 and own_f32(n, 4 * C, C, ends=True)
        self.f = None if self.fused_ffn or self.own_ffn1 else buf(n, 4 * C)
        # norm factors of committed depth-mix candidates, carried from mix to mix (16-byte rows needed)
        self.cache_norms = CACHE_NORMS and (C * emb.element_size()) % 16 == 0
        self.norm_cache: dict[int, torch.Tensor] = {}
        self.prefix_o = None
        self.prefix_lse = None
        self.part_o = None
        self.part_lse = None
        self.prefix_on_tc = False
        self.prefix_ctas = 0
        self.workspace = None

    def _mix(self, cands: list, partial: torch.Tensor, w: torch.Tensor, known: set) -> None:
        """Depth mix of the committed candidates and the running block sum into self.u.  A committed candidate no
        longer changes, so the first mix that sees it writes its per-row norm factor and the later ones read it."""
        if not self.cache_norms:
            ops.depthmix(cands + [partial], w, None, self.u)
            return
        inv_in, inv_out, out_index = [], None, -1
        for idx, t in enumerate(cands):
            key = t.data_ptr()
            if key in known:
                inv_in.append(self.norm_cache[key])
            else:
                inv_in.append(None)
                if inv_out is None and not any(c.data_ptr() == key for c in cands[:idx]):
                    buf = self.norm_cache.get(key)
                    if buf is None:
                        buf = self.norm_cache[key] = torch.empty(self.n, dtype=torch.float32, device=t.device)
                    inv_out, out_index = buf, idx
        ops.depthmix_cached(cands + [partial], inv_in + [None], w, None, self.u, inv_out, out_index)
        if inv_out is not None:
            known.add(cands[out_index].data_ptr())

    def _linear(self, a: torch.Tensor, w_t: torch.Tensor, out: torch.Tensor, name: str, add: bool = False) -> None:
        """out (+)= a @ w_t: a small fp32 model's and a lone bf16 row on the library's kernels, others on cuBLAS."""
        if self.f32 and own_f32(out.shape[0], out.shape[1], a.shape[1], ends=add):
            ops.linear_f32(a, w_t.t(), out, add=out if add else None)
            return
        if self.one_row:
            ops.linear(a, w_t.t(), out, add=out if add else None, status=self.status)
            return
        with region(name):
            if add:
                out.addmm_(a, w_t)
            else:
                torch.mm(a, w_t, out=out)

    def _decode_extras(self, b: KvBinding) -> None:
        m = self.model
        H, D = m.n_head, m.n_embd // m.n_head
        dev = self.x.device
        if b.shared_layouts is not None and self.prefix_o is None:
            self.prefix_o = torch.empty((self.n, H, D), dtype=torch.float32, device=dev)
            self.prefix_lse = torch.empty((self.n, H), dtype=torch.float32, device=dev)
        if b.shared_layouts is not None and b.overlap_prefix and b.n_splits == 1 and self.part_o is None:
            self.part_o = torch.empty((self.n, H, D), dtype=torch.float32, device=dev)
            self.part_lse = torch.empty((self.n, H), dtype=torch.float32, device=dev)
            self.side = torch.cuda.Stream(device=dev, priority=SIDE_PRIORITY)
            n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
            rows, size = b.rows_per_series, self.q.element_size()
            units = (self.n // rows) * H * (-(-rows // 256))
            # the per-row phase: its bytes at the copy rate, and what a warp per (row, head) costs however few its keys
            own_us = self.n * H * (2 * D * size * b.own_keys / 6.65e6 + 4e-4)
            self.prefix_ctas = prefix_ctas(units, -(-b.shared_keys // 128), own_us, n_sm)
            # the persistent tensor-core kernel covers bf16 heads of 32, 64 or 128 in pages that tile its 128-key
            # blocks; other models leave the choice to the library (its warp-level kernel)
            pt = int(b.shared_layouts[0].page_tokens)
            self.prefix_on_tc = (
                self.q.dtype == torch.bfloat16 and D in (32, 64, 128) and pt >= 8 and (pt % 128 == 0 or 128 % pt == 0)
            )
        if b.n_splits > 1 and self.workspace is None:
            nbytes = ops.decode_attn_workspace_bytes(self.n, H, D, b.n_splits)
            self.workspace = torch.empty(nbytes // 4, dtype=torch.float32, device=dev)

    def run_whole(self, ids32: torch.Tensor, b: KvBinding, n_steps: int = 1, draw=None) -> torch.Tensor:
        """The forward in one launch (`whole`), or `n_steps` decode steps with their draws."""
        first = b.layouts[0]
        stride = (b.layouts[1].k_base - first.k_base) // 4 if len(b.layouts) > 1 else 0
        decode = {"len0": b.len0, "start1": b.start1, "len1": b.len1} if b.decode else {"T": self.T, "last_only": self.last_only}
        ops.small_gpt(
            self.model.packed_weights().whole(self.model), first, stride, ids32, b.pos0, b.slot0, b.step, self.logits, self.status,
            max_keys=self.keys, logit_cap=self.cap, n_steps=n_steps, draw=draw, **decode,
        )
        return self.logits

    def run(self, ids32: torch.Tensor, b: KvBinding) -> torch.Tensor | None:
        if self.whole:
            return self.run_whole(ids32, b)
        m = self.model
        C, H, L = m.n_embd, m.n_head, m.n_layer
        D = C // H
        T, n_seq = self.T, self.n_seq
        W = m.packed_weights()
        if b.decode:
            assert T == 1
            self._decode_extras(b)
        ops.embed_rmsnorm(ids32, W.emb, self.x)
        cands = [self.x]
        partial = self.x
        known: set[int] = set()  # committed candidates whose norm factor has been written during this forward
        for i in range(L):
            lw = W.layers[i]
            if i == 0:
                ops.depthmix([self.x], None, None, self.u)  # single candidate: mix is the identity
            else:
                self._mix(cands, partial, lw.w_attn, known)
            if (i + 1) % m.attn_res_layers_per_block == 0:
                cands = cands + [partial]
                partial = None
            self._linear(self.u, lw.wqkvg_t, self.qkvg, "gemm_qkvg")
            qv, kv_, vv, gv = (self.qkvg[:, j * C : (j + 1) * C] for j in range(4))
            ops.rope_qknorm_kvappend(
                qv, kv_, vv, self.q, W.freqs_cis, b.layouts[i], b.pos0, b.slot0, b.step, n_seq, T, H, D, self.status
            )
            if b.decode:
                po = pl = None
                if b.shared_layouts is not None:
                    N = b.rows_per_series
                    prefix_phase = lambda: ops.fmha_prefill(  # noqa: E731
                        self.q, b.shared_layouts[i], self.prefix_o, B=n_seq // N, H=H, Tq=N, D=D,
                        q_batch_stride=N * C, q_row_stride=C, o_batch_stride=N * C, o_row_stride=C,
                        kv_len=b.shared_len, causal=False, lse=self.prefix_lse,
                        impl=PREFIX_IMPL if (self.side is not None and PREFIX_IMPL and self.prefix_on_tc) else b.fmha_impl,
                        status=self.status,
                        max_ctas=self.prefix_ctas if self.side is not None else 0,
                    )
                    po, pl = self.prefix_o, self.prefix_lse
                if po is not None and self.side is not None:
                    # The tensor-core contraction over the shared prompt and the HBM-bound pass over each
                    # row's own tokens need different parts of the SM: run them side by side, then merge.
                    main = torch.cuda.current_stream()
                    self.side.wait_stream(main)
                    with torch.cuda.stream(self.side):
                        prefix_phase()
                    ops.decode_attn_partial(
                        self.q, b.layouts[i], None, b.start1, b.len1, b.step, self.part_o, self.part_lse, H=H, D=D
                    )
                    main.wait_stream(self.side)
                    ops.attn_merge(po, pl, self.part_o, self.part_lse, self.y, H=H, D=D, gate=gv)
                else:
                    if po is not None:
                        prefix_phase()
                    ops.decode_attn(
                        self.q, b.layouts[i], b.len0, b.start1, b.len1, b.step, self.y, H=H, D=D, gate=gv,
                        prefix_o=po, prefix_lse=pl, workspace=self.workspace, n_splits=b.n_splits,
                    )
            else:
                own_gate = b.fmha_impl != 4  # the kernel with two query tiles per CTA is not built with one
                ops.fmha_prefill(
                    self.q, b.layouts[i], self.y, B=n_seq, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C,
                    o_batch_stride=T * C, o_row_stride=C, kv_len_all=b.kv_len, q_offset=b.q_offset, causal=True,
                    impl=b.fmha_impl, status=self.status, gate=gv if own_gate else None,
                )
                if not own_gate:
                    ops.sigmoid_gate(self.y, gv)
            part = self.parts[i]
            if partial is None:
                self._linear(self.y, lw.wproj_t, part, "gemm_proj")
            else:  # layers_per_block > 1: the running block sum keeps accumulating
                with region("gemm_proj"):
                    torch.addmm(partial, self.y, lw.wproj_t, out=part)
            partial = part
            self._mix(cands, partial, lw.w_mlp, known)
            if self.fused_ffn:  # first FFN GEMM with the SwiGLU in its epilogue (the [n, 4C] product never reaches HBM)
                ops.linear(self.u, lw.w1, self.act, swiglu=(m.swiglu_alpha, m.swiglu_limit), status=self.status)
            elif self.own_ffn1:
                ops.linear_f32(self.u, lw.w1, self.act, swiglu=(m.swiglu_alpha, m.swiglu_limit))
            else:
                with region("gemm_ffn1"):
                    torch.mm(self.u, lw.w1_t, out=self.f)
                ops.swiglu(self.f, self.act, m.swiglu_alpha, m.swiglu_limit)
            # bf16 on cuBLAS: 6.6 / 9.8 us for the two n_embd-wide GEMMs of 4096 rows against 9.5 / 14.4 us for dgpt_linear
            self._linear(self.act, lw.w2_t, partial, "gemm_ffn2", add=True)
        final = partial
        if self.last is not None:
            self.last.copy_(partial.view(n_seq, T, C)[:, T - 1, :])
            final = self.last
        ops.depthmix([final], None, None, self.xn)
        if self.logits is None:
            return None
        if self.own_head:
            ops.linear(self.xn, W.emb, self.logits, softcap=self.cap, tiles=not self.few_rows, status=self.status)
        elif self.f32 and own_f32(*self.logits.shape, C, ends=self.cap > 0):
            ops.linear_f32(self.xn, W.emb, self.logits, softcap=self.cap)
        else:
            with region("gemm_logits"):
                torch.mm(self.xn, W.emb.t(), out=self.logits)
            if self.cap > 0:
                ops.softcap_(self.logits, self.cap)
        return self.logits


@dataclass
class _LayerWeights:
    w1: torch.Tensor
    wqkvg_t: torch.Tensor
    wproj_t: torch.Tensor
    w1_t: torch.Tensor
    w2_t: torch.Tensor
    w_attn: torch.Tensor
    w_mlp: torch.Tensor


@dataclass
class _Packed:
    emb: torch.Tensor
    freqs_cis: torch.Tensor
    layers: list
    rows16: bool  # every matrix lies as the linear kernels want it
    stamp: tuple
    columns: torch.Tensor | None  # the same weights as dgpt_small_gpt reads them, where it is built for the model

    def whole(self, m: "GPT"):
        return ops.small_gpt_model(
            self.emb, self.columns, self.freqs_cis, H=m.n_head, L=m.n_layer, layers_per_block=m.attn_res_layers_per_block,
            swiglu=(m.swiglu_alpha, m.swiglu_limit),
        )

    @property
    def head(self) -> torch.Tensor:
        return self.emb


def _parameters(module: nn.Module) -> list:
    """Every parameter in the tree as it is now, a tied one as often as it occurs.  (`parameters()` names and compares them on its way:
    50 us a call for 2 layers, which a recorded token pays every time.)"""
    found, below = [], [module]
    while below:
        m = below.pop()
        found += [p for p in m._parameters.values() if p is not None]
        below += [c for c in m._modules.values() if c is not None]
    return found


def _small_gpt_columns(layers: list, emb: torch.Tensor) -> torch.Tensor:
    """Weights of all layers and the head as dgpt_small_gpt reads them (see include/dgpt.h)."""

    def words(w: torch.Tensor) -> torch.Tensor:  # [N, K] -> [K / 4 / S][N][S][4]
        N, K = w.shape
        S = max(1, min(256 // N, K // 4))
        return w.reshape(N, K // 4 // S, S, 4).transpose(0, 1).reshape(-1)

    flat = [words(w) for l in layers for w in (l.wqkvg_t.t(), l.wproj_t.t(), l.w1, l.w2_t.t())]
    flat += [words(F.pad(rows, (0, 0, 0, 256 - rows.shape[0]))) for rows in emb.split(256)]
    return torch.cat(flat + [v for l in layers for v in (l.w_attn, l.w_mlp)])


class GPT(DeviceModel):
    def __init__(
        self,
        vocab_size: int,
        n_embd: int = 64,
        block_size: int = 32,
        n_head: int = 4,
        n_layer: int = 4,
        rope_theta: float = 10000,
        swiglu_alpha: float = 1.702,
        swiglu_limit: float = 7.0,
        use_checkpoint: bool = True,
        logit_softcap: float = 15.0,
        pad_vocab_size_to: int = 64,
        attn_res_layers_per_block: int = 1,
        label_smoothing_sigma: float = 0.0,
    ) -> None:
        super().__init__(block_size=block_size, vocab_size=vocab_size, n_embd=n_embd, n_head=n_head, n_layer=n_layer)
        assert logit_softcap >= 0, "logit_softcap must be non-negative (0 disables it)"
        assert label_smoothing_sigma >= 0, "label_smoothing_sigma must be non-negative (0 disables it)"
        assert pad_vocab_size_to >= 1, "pad_vocab_size_to must be >= 1"
        assert attn_res_layers_per_block >= 1, "attn_res_layers_per_block must be >= 1"
        assert vocab_size % pad_vocab_size_to == 0, (
            f"vocab_size ({vocab_size}) must be a multiple of "
            f"pad_vocab_size_to ({pad_vocab_size_to}); pad it in the encoder"
        )
        self.token_embedding_table = nn.Embedding(vocab_size, n_embd)
        self.blocks = nn.ModuleList(
            Block(n_embd, n_head, swiglu_alpha, swiglu_limit, layer_idx=i, layers_per_block=attn_res_layers_per_block)
            for i in range(n_layer)
        )
        self.lm_head = nn.Linear(n_embd, vocab_size, bias=False)
        self.lm_head.weight = self.token_embedding_table.weight  # tied
        self.register_buffer(
            "freqs_cis", precompute_freqs_cis(n_embd // n_head, block_size * 2, theta=rope_theta), persistent=False
        )
        self.use_checkpoint = use_checkpoint
        self.logit_softcap = logit_softcap
        self.label_smoothing_sigma = label_smoothing_sigma
        self.swiglu_alpha = swiglu_alpha
        self.swiglu_limit = swiglu_limit
        self.attn_res_layers_per_block = attn_res_layers_per_block
        self._packed: _Packed | None = None

    def report(self) -> torch.Tensor | None:
        if self.late_status is None:
            self.late_status = LateStatus()
        return self.late_status.word()

    # ---- weights as the kernels want them -------------------------------------------
    def packed_weights(self) -> _Packed:
        """Fused QKVG weight and transposed views, rebuilt when a parameter was modified or moved."""
        stamp = tuple([(p.data_ptr(), p._version, p.dtype) for p in _parameters(self)]) + (self.freqs_cis.data_ptr(),)
        if self._packed is not None and self._packed.stamp == stamp:
            return self._packed
        layers = []
        with torch.no_grad():
            for blk in self.blocks:
                a = blk.sa
                wqkvg = torch.cat([a.c_q.weight, a.c_k.weight, a.c_v.weight, a.c_g.weight], dim=0).contiguous()
                layers.append(
                    _LayerWeights(
                        w1=blk.ffwd.net[0].weight.detach(),
                        wqkvg_t=wqkvg.t(),
                        wproj_t=a.c_proj.weight.detach().t(),
                        w1_t=blk.ffwd.net[0].weight.detach().t(),
                        w2_t=blk.ffwd.net[2].weight.detach().t(),
                        w_attn=blk.attn_res_proj.weight.detach().reshape(-1),
                        w_mlp=blk.mlp_res_proj.weight.detach().reshape(-1),
                    )
                )
            emb = self.token_embedding_table.weight.detach()
            table = self.freqs_cis.to(emb.dtype).contiguous()
            columns = None
            if emb.dtype == torch.float32 and ops.small_gpt_supported(self.n_embd, self.n_head, self.n_layer, self.vocab_size):
                columns = _small_gpt_columns(layers, emb)
        rows16 = ops.rows16(emb) and all(ops.rows16(w) for l in layers for w in (l.w1, l.wproj_t.t(), l.w2_t.t()))
        self._packed = _Packed(emb=emb, freqs_cis=table, layers=layers, rows16=rows16, stamp=stamp, columns=columns)
        return self._packed

    @classmethod
    def from_config(cls, config: dict) -> "GPT":
        """The constructor's keywords as a configuration."""
        return cls(**{k: v for k, v in config.items() if k != "architecture"})

    def load_tensors(self, tensors: dict) -> None:
        """A checkpoint under the state_dict names; the tied head may be left out."""
        tensors = dict(tensors)
        tensors.setdefault("lm_head.weight", tensors["token_embedding_table.weight"])
        self.load_state_dict(tensors)

    # ---- what the Engine needs ----------------------------------------------------------
    @property
    def embedding(self) -> torch.Tensor:
        return self.token_embedding_table.weight

    def new_cache(self, batch_size: int = 1, seq_len: int = 0) -> KVCache:
        return KVCache(batch_size=batch_size, num_heads=self.n_head, seq_len=max(seq_len, 1),
                       head_dim=self.n_embd // self.n_head, num_layers=self.n_layer)

    def cache_storage(self, cache: KVCache) -> tuple:
        return (cache.kv_cache,)

    @torch.inference_mode()
    def logits_at(self, idx: torch.Tensor, cache: KVCache, rows: torch.Tensor) -> torch.Tensor:
        return self(idx, kv_cache=cache)[0][0].index_select(0, rows)

    def single_step(self, cache: KVCache, old: SingleStep | None, stream: torch.cuda.Stream) -> SingleStep | None:
        t0, H, emb = cache.get_pos(), self.n_head, self.embedding
        if t0 == 0:
            return None
        assert t0 + 1 <= self.freqs_cis.shape[0]
        cache.ensure(t0 + 1, emb.dtype, emb.device)
        splits = _pick_splits(H, t0 + 1)
        keys = -(-(t0 + 1) // 256) * 256  # a plan serves many tokens
        whole = whole_f32(self.n_embd, H, self.n_layer, self.vocab_size, 1, 1, keys) and keys
        kind = (splits, whole, self.logit_softcap, self.swiglu_alpha, self.swiglu_limit, self.attn_res_layers_per_block)
        held = (self.packed_weights(), *self.cache_storage(cache))
        if old is not None and old.fits(kind, held):
            return old
        with torch.cuda.stream(stream):
            numbers = torch.zeros(4, dtype=torch.int32, device=emb.device)
            zero = torch.zeros(1, dtype=torch.int32, device=emb.device)
            bind = KvBinding(
                layouts=[cache.layer_layout(i) for i in range(self.n_layer)], pos0=numbers[2:3], slot0=numbers[1:2], decode=True,
                len0=zero, start1=zero, len1=numbers[3:4], n_splits=splits,
            )
            return SingleStep(ForwardPlan(self, 1, 1, cap=self.logit_softcap, keys=keys, late=True), bind, numbers, kind, held, checks=False)

    def paged_cache(self, n_series, rows_per_series, prefix_len, max_new, page_tokens, pool=None) -> PagedKVCache:
        emb = self.embedding
        return PagedKVCache(self.n_layer, self.n_head, self.n_embd // self.n_head, n_series, rows_per_series, prefix_len, max_new,
                            emb.dtype, emb.device, page_tokens=page_tokens, pool=pool)

    def prefill_plan(self, cache, members, P, fmha_impl, few_rows=True):
        idx = torch.tensor(members, device=cache.prefix_table.device)
        table = cache.prefix_table[idx].contiguous()
        zero = torch.zeros(len(members), dtype=torch.int32, device=table.device)
        bind = KvBinding(
            layouts=[cache._layout(l, table) for l in range(self.n_layer)], pos0=zero, slot0=zero, kv_len=P, q_offset=0,
            fmha_impl=fmha_impl,
        )
        return bind, ForwardPlan(self, len(members), P, last_only=True, few_rows=few_rows, keys=None if fmha_impl else P)

    def decode_plan(self, cache, prompt_lens, max_keys, step, shared, fmha_impl, overlap_prefix, want_logits, few_rows=True):
        R, L = cache.n_rows, self.n_layer
        row_len = prompt_lens.repeat_interleave(cache.rows_per_series)
        slot0 = torch.full((R,), cache.suffix_slot0, dtype=torch.int32, device=row_len.device)
        bind = KvBinding(
            layouts=[cache.row_layout(l) for l in range(L)],
            pos0=row_len.contiguous(),
            slot0=slot0,
            step=step,
            decode=True,
            len0=row_len.contiguous(),
            start1=slot0,
            len1=torch.ones(R, dtype=torch.int32, device=row_len.device),
            n_splits=1 if shared else _pick_splits(R * self.n_head, max_keys),
            shared_layouts=[cache.prefix_layout(l) for l in range(L)] if shared else None,
            shared_len=prompt_lens if shared else None,
            shared_keys=cache.prefix_len,
            own_keys=max(1, cache.max_new // 2),
            rows_per_series=cache.rows_per_series,
            fmha_impl=fmha_impl,
            overlap_prefix=overlap_prefix and shared,
        )
        return bind, ForwardPlan(self, R, 1, want_logits=want_logits, few_rows=few_rows, keys=None if fmha_impl else max_keys)

    # ---- the reference contract --------------------------------------------------------
    def forward(
        self,
        idx: torch.Tensor,
        targets: torch.Tensor | None = None,
        kv_cache: KVCache | None = None,
    ) -> tuple[torch.Tensor, torch.Tensor | None]:
        if not idx.is_cuda:
            raise RuntimeError("diff_gpt_b200.GPT runs on CUDA only; there is no CPU path")
        if torch.is_grad_enabled() and any(p.requires_grad for p in self.parameters()) and self.training:
            raise NotImplementedError("training (backward) is outside this build; use the reference module to train")
        with torch.no_grad():
            logits = self._infer(idx, kv_cache)
        loss = None
        if targets is not None:
            flat, tgt = logits.view(-1, logits.shape[-1]).float(), targets.view(-1)
            if self.label_smoothing_sigma > 0:
                loss = _ordinal_soft_ce(flat, tgt, self.label_smoothing_sigma)
            else:
                loss = F.cross_entropy(flat, tgt)
        return logits, loss

    def _infer(self, idx: torch.Tensor, kv_cache: KVCache | None) -> torch.Tensor:
        B, T = idx.shape
        C, H, L, V = self.n_embd, self.n_head, self.n_layer, self.vocab_size
        D = C // H
        dev = idx.device
        dt = self.token_embedding_table.weight.dtype
        t0 = 0 if kv_cache is None else kv_cache.get_pos()
        assert t0 + T <= self.freqs_cis.shape[0]
        if self.late_status is not None:
            self.late_status.check()
        plan = ForwardPlan(self, B, T, cap=self.logit_softcap, keys=t0 + T, late=True)
        if kv_cache is None:
            # every layer reuses the same scratch K/V, unless one kernel's CTAs work on different layers at one time
            scratch = KVCache(batch_size=B, num_heads=H, seq_len=T, head_dim=D, num_layers=L if plan.whole else 1)
            scratch.ensure(T, dt, dev)
            layouts = [scratch.layer_layout(i if plan.whole else 0) for i in range(L)]
        else:
            assert not isinstance(kv_cache, PagedKVCache), "PagedKVCache is driven by the Engine"
            kv_cache.ensure(t0 + T, dt, dev)
            layouts = [kv_cache.layer_layout(i) for i in range(L)]
        start = torch.full((B,), t0, dtype=torch.int32, device=dev)
        bind = KvBinding(layouts=layouts, pos0=start, slot0=start, kv_len=t0 + T, q_offset=t0)
        if T == 1 and t0 > 0:
            zeros = torch.zeros(B, dtype=torch.int32, device=dev)
            bind.decode = True
            bind.len0, bind.start1 = zeros, zeros
            bind.len1 = torch.full((B,), t0 + 1, dtype=torch.int32, device=dev)
            n_keys = t0 + 1
            bind.n_splits = _pick_splits(B * H, n_keys)
        logits = plan.run(idx.reshape(-1).to(torch.int32), bind)
        if kv_cache is not None:
            kv_cache.pos = t0 + T
        return logits.view(B, T, V)

    @torch.inference_mode()
    def generate(self, idx: torch.Tensor, max_new_tokens: int, sampler: Sampler | None, seed: int | None = None):
        """Naive sliding-window generation without a cache (gpt.py:202-237); kept for API parity."""
        rng = None
        if seed is not None:
            rng = torch.Generator(device=idx.device)
            rng.manual_seed(seed)
        B, T = idx.shape
        out = torch.zeros((B, T + max_new_tokens), dtype=torch.int64, device=idx.device)
        out[:, :T] = idx
        for cur in range(T, T + max_new_tokens):
            window = out[:, max(0, cur - self.block_size) : cur]
            logits = self(window)[0][:, -1]
            if sampler is not None:
                nxt = sampler(logits, rng=rng)
            else:
                nxt = torch.multinomial(F.softmax(logits.float(), dim=-1), num_samples=1, generator=rng)
            out[:, cur] = nxt.reshape(-1)
        return out

    @property
    def device_type(self) -> str:
        return str(self.freqs_cis.device.type)


GPT.step_path = ((GPT, "logits_at"), (nn.Module, "__call__"), (GPT, "forward"), (GPT, "_infer"))

_SM_COUNT: dict[int, int] = {}


def _sm_count() -> int:
    """Multiprocessors of the current CUDA device (148 on a B200); that figure is assumed where no device is present,
    so the split policy can be examined on a CPU box."""
    dev = torch._C._cuda_getDevice() if torch.cuda.is_initialized() else -1
    if dev not in _SM_COUNT:
        if not torch.cuda.is_available():
            return 148
        dev = torch.cuda.current_device()
        _SM_COUNT[dev] = torch.cuda.get_device_properties(dev).multi_processor_count
    return _SM_COUNT[dev]


def _pick_splits(n_pairs: int, n_keys: int) -> int:
    """Split the keys when (row, head) pairs alone cannot fill the GPU: as many splits as leave one wave of CTAs, 16 warps on
    every multiprocessor.  One more split makes a second wave of a few CTAs: 64 rows, 8 heads of 64, 3682 keys, us: 4 splits (512
    CTAs of 592) 76, 5 splits (640) 96; 130 rows, 1400 keys: 2 splits 61, 3 splits 71."""
    room = _sm_count() * 16
    if n_pairs <= 0 or 2 * n_pairs > room or n_keys < 512:
        return 1
    return max(1, min(room // n_pairs, n_keys // 256, 64))


def _ordinal_soft_ce(logits: torch.Tensor, targets: torch.Tensor, sigma: float, ignore_index: int = -100):
    """Cross entropy against a Gaussian bump of width sigma (in bins) centred on the target bin."""
    keep = targets != ignore_index
    if not bool(keep.any()):
        return logits.sum() * 0.0
    lg, tg = logits[keep], targets[keep]
    bins = torch.arange(lg.shape[-1], device=lg.device, dtype=lg.dtype)
    soft = F.softmax(-((bins[None, :] - tg[:, None].to(lg.dtype)) ** 2) / (2.0 * sigma * sigma), dim=-1)
    return -(soft * F.log_softmax(lg, dim=-1)).sum(dim=-1).mean()
