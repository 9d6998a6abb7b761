"""The step function: model, cache and kernels behind one call.

``ModelRunner.step(entries)`` runs exactly the tokens it is given, as one
batch, from the cache that earlier steps left, and returns the logits at the
wanted places.  Generation, the scheduler and trace replay all go through it.
The reference's counterpart is execute_model_step -> forward_packed
(crates/vllm-engine/src/engine.rs:175-286,
crates/vllm-models/src/llama/architecture.rs:141-156).

How a step reaches the GPU: steps of single tokens replay a CUDA graph over a
static batch (``decode_step_flat``; the graph copies its inputs in, chooses
the tokens and copies them out), and the step after such a step can be
launched before its tokens are known (``decode_follow``); other steps whose
packed layout repeats replay a graph captured for that layout
(``_step_shape_graph``); everything else launches its kernels one by one.
"""
from __future__ import annotations

import contextlib
import dataclasses
import gc
import os

import numpy as np
import torch

from ..cache.manager import CacheManager
from ..config.registry import load_config
from ..parts.base import CacheView
from ..parts.model import DecoderModel, TensorBank, expected_tensors
from ..parts.spec import BuildEnv
from ..weights.loader import load_weights
from .. import ops
from ..cache.manager import CacheError
from .batch import BatchError, StepBatch, StepEntry, build_step_batch

_DTYPES = {"bfloat16": torch.bfloat16, "bf16": torch.bfloat16, "float32": torch.float32, "fp32": torch.float32,
           "f32": torch.float32}


# Steps other than single tokens' (which have graphs of their own) go through a graph captured for their layout once that
# layout repeats: a portion's size is mostly the scheduler's, and the step of a prompt's next portion beside the same decoding
# requests has the layout of the one before.  From SHAPE_GRAPH_MIN_TOKENS tokens on at the second step of a layout; shorter
# steps at the SMALL_GRAPH_AT-th: what a replay saves there is host time (some 30 to 85 launches of 14 to 18 us), a capture
# costs as much as some of them, and short prompts' layouts are many.  So many layouts of either kind are kept.  Where more
# of them come in turn than are kept, a short step's graph gives way only once it has not been used for so many steps: every
# step would cost a capture otherwise (RepeatedLayouts).  Long ones, whose captures cost a step or two, give way at once.
SHAPE_GRAPH_MIN_TOKENS = 256
SHAPE_GRAPHS_KEPT = 4
SMALL_GRAPH_AT = 4
SMALL_GRAPHS_KEPT = 16
GIVES_WAY_AFTER = 0, 1024          # steps without use: graphs of long steps, of short ones
# Steps of single tokens have a graph for each power of two of the longest context from 1,024 on, and one for contexts of up to
# SHORT_CONTEXT: attention in one part (at 1,024 keys in four), so that no kernel adds parts up.  60 keys each, us a step: the 1B model
# 1 request 641 to 606, 8 678 to 636, 32 910 to 857; kasarax's sizes 198 to 194, 207 to 202, 327 to 316.  At 200 keys the 1B model
# still gains (637 to 626, 675 to 656, 908 to 875), kasarax loses (198 to 203, 208 to 210); at 400 keys
# both lose up to 8 requests (643 to 652; 198 to 212).
SHORT_CONTEXT = 128
LAYOUTS_COUNTED = 64, 512          # layouts whose steps are counted: of long steps, of short ones


@contextlib.contextmanager
def capture(graph):
    """``torch.cuda.graph(graph)`` with Python's cyclic garbage collector held off: a collection in the middle of
    a capture may free a page-locked host buffer of an earlier step, and freeing one records an event on the
    stream that used it, which is not allowed on a capturing stream and invalidates the capture."""
    was_enabled = gc.isenabled()
    gc.disable()
    try:
        with torch.cuda.graph(graph):
            yield
    finally:
        if was_enabled:
            gc.enable()


def raise_device_error(code: int):
    """What a kernel left in an error flag: 1 for a position outside its table."""
    if code == 1:
        raise RuntimeError("a kernel met a position outside its table")
    raise RuntimeError(f"a kernel flagged error {code}; the step's result is invalid")


# RAILGUN_B200_NVTX=1 puts a named range around every step (visible in a profiler's timeline).
NVTX = os.environ.get("RAILGUN_B200_NVTX", "0") == "1"


def parse_dtype(name):
    if isinstance(name, torch.dtype):
        if name not in (torch.bfloat16, torch.float32):
            raise ValueError(f"dtype {name} is not supported: bfloat16 or float32")
        return name
    try:
        return _DTYPES[str(name).lower()]
    except KeyError:
        raise ValueError(f"dtype {name!r} is not supported: bfloat16 or float32") from None


class _CacheViews:
    def __init__(self, cache: CacheManager):
        self._views = {}
        for cid, t in cache.kv.items():
            self._views[cid] = CacheView(cid, group=cache.group_of[cid], kv=t, page_size=cache.page_size_of(cid))
        for cid, t in cache.state.items():
            self._views[cid] = CacheView(cid, state=t)
        # a mixer that asked for a tuple of needs sees one view per need
        for cid, n in cache.composite.items():
            self._views[cid] = CacheView(cid, parts=tuple(self._views.get((cid, k)) or CacheView(cid)
                                                          for k in range(n)))
        self._none = {}

    def view(self, cid):
        v = self._views.get(cid)
        if v is None:
            v = self._none.setdefault(cid, CacheView(cid))
        return v


def build_model(model_dir, dtype, device, spec_override=None):
    """Read config.json, pick the architecture from the registry, load the
    weights by name and build the model.  Returns (architecture, config, model)."""
    arch, cfg = load_config(model_dir)
    spec = spec_override(cfg) if spec_override else arch.model_spec(cfg)
    expected = expected_tensors(spec)
    tensors = load_weights(model_dir, expected, device="cpu", allow_unexpected=arch.allow_unexpected(cfg))
    env = BuildEnv(device=device, dtype=dtype, hidden_size=spec.hidden_size, max_position=spec.max_position)
    model = DecoderModel(spec, env, TensorBank(tensors, device))
    return arch, cfg, model


_BATCH_BUCKETS = (1, 2, 4, 8, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)


def _bucket(n: int, buckets) -> int:
    for b in buckets:
        if n <= b:
            return b
    return n


class StaticDecodeBatch:
    """Device buffers of fixed address for decode steps of up to ``B`` requests
    whose contexts stay within ``MB`` pages, with the pinned host buffer that
    is copied into them in one transfer.  A graph captured over these buffers
    can be replayed for any such step.  Layout (int32): token ids | positions |
    context lengths | start positions | state slots | per group slot mapping |
    per group block table [B, MB] | the rows' sampling parameters (seed and
    draw counter as 64-bit, temperature, top-k, top-p)."""

    def __init__(self, runner, B: int, MB: int):
        dev = runner.device
        G = len(runner.page_sizes)
        self.B, self.MB, self.G = B, MB, G
        self.sampling_off = -(-((5 + G) * B + G * B * MB) // 2) * 2          # even: 64-bit values start there
        n_ints = self.sampling_off + 7 * B
        self.host = torch.zeros(n_ints, dtype=torch.int32, pin_memory=True)
        self.host_np = self.host.numpy()
        # the step's tokens and, behind them, the flag that a kernel raises for a position outside its table:
        # one copy by the graph brings both to the host
        self.host_out = torch.zeros(B + 1, dtype=torch.int32, pin_memory=True)
        self.host_out_np = self.host_out.numpy()
        self.out_dev = torch.zeros(B + 1, dtype=torch.int32, device=dev)
        self.dev = torch.zeros(n_ints, dtype=torch.int32, device=dev)
        seg = lambda i: self.dev[i * B:(i + 1) * B]
        ar = torch.arange(B + 1, dtype=torch.int32, device=dev)
        tables_off = (5 + G) * B
        self.batch = StepBatch(
            num_tokens=B, num_requests=B, num_wanted=B, max_query_len=1,
            max_context_len=MB * (min(runner.page_sizes) if G else 1),
            token_ids=seg(0), positions=seg(1), req_of_token=ar[:B], want_rows=ar[:B], cu_seqlens=ar,
            context_lens=seg(2), start_pos=seg(3), state_slots=seg(4),
            slot_mapping=[seg(5 + g) for g in range(G)],
            block_table=[self.dev[tables_off + g * B * MB:tables_off + (g + 1) * B * MB].view(B, MB)
                         for g in range(G)],
            err_flag=self.out_dev[B:], decode_only=True)
        self.sampling = sampling_views(self.dev, self.sampling_off, B)        # device views of the sampling parameters
        self.sampled = self.out_dev[:B]                                         # the tokens the last step chose
        self.step_graphs = {}          # with sampling parameters or greedy -> CapturedStep
        self.follow = [None, None]     # FollowStep: the same step fed with ``sampled`` instead of host tokens
        self.in_flight = None          # an event after the last replay, which writes ``host_out``
        self.stream = self.stream_handle = None     # the stream that its last step was launched on
        # the number of the step last packed into ``host`` and of the one whose step has read it (written by that step)
        self.seq = torch.zeros(2, dtype=torch.int32, pin_memory=True)
        self.seq_np = self.seq.numpy()
        self.blocks_done = torch.zeros(2, dtype=torch.int32, device=dev)

    def raise_if_flagged(self, host_out_np) -> None:
        code = int(host_out_np[self.B])
        if code:
            self.out_dev[self.B:].zero_()
            host_out_np[self.B] = 0
            raise_device_error(code)

    def wait_until_reusable(self) -> None:
        """``host`` may be written again once the last step packed into it has read it: its first kernel says so, while
        the rest of the step still runs."""
        while self.in_flight is not None and self.seq_np[1] != self.seq_np[0]:
            if self.in_flight.query():                       # the step is over (raises if it failed)
                break

    def packed(self) -> None:
        """``host`` holds another step: number it, for ``wait_until_reusable``."""
        self.seq_np[0] = (int(self.seq_np[0]) + 1) & 0x7fffffff


def sampling_views(buf, off: int, B: int) -> dict:
    """The sampling parameters inside a packed decode buffer (a torch tensor or a numpy array of int32)."""
    f32, i64 = (torch.float32, torch.int64) if isinstance(buf, torch.Tensor) else (np.float32, np.int64)
    return dict(seed=buf[off:off + 2 * B].view(i64), counter=buf[off + 2 * B:off + 4 * B].view(i64),
                temperature=buf[off + 4 * B:off + 5 * B].view(f32), top_k=buf[off + 5 * B:off + 6 * B],
                top_p=buf[off + 6 * B:off + 7 * B].view(f32))


class FollowStep:
    """A decode step launched before the tokens of the step before it are on the
    host: its graph takes positions, slots and block tables from this object's
    own pinned buffer, the token ids from the static batch's ``sampled``, and
    copies its greedy tokens into this object's pinned ``host_out``.  Two of
    them alternate per static batch, so that a step in flight never shares a
    pinned buffer with the step that is being read."""

    def __init__(self, static: StaticDecodeBatch):
        self.static = static
        self.host_in = torch.zeros(static.host.numel(), dtype=torch.int32, pin_memory=True)
        self.host_in_np = self.host_in.numpy()
        self.host_out = torch.zeros(static.B + 1, dtype=torch.int32, pin_memory=True)
        self.host_out_np = self.host_out.numpy()
        self.done = torch.cuda.Event()
        self.captured = {}             # with sampling parameters or greedy -> CapturedStep
        self.ids = None                # the requests of the launched step, in row order

    def tokens(self) -> np.ndarray:
        """The launched step's tokens, one per row (waits for the step; raises if a kernel of it flagged an error)."""
        self.done.synchronize()
        self.static.raise_if_flagged(self.host_out_np)
        return self.host_out_np[:self.static.B]


class ShapeGraph:
    """A captured step for one packed layout: the static device buffer the step's
    data is copied into, the batch whose tensors are views of it, the graph and
    its output."""

    def __init__(self, dev, batch, graph, logits, launches):
        self.dev, self.batch, self.graph, self.logits, self.launches = dev, batch, graph, logits, launches
        self.hold = None               # the last packed step (keeps its pinned buffer alive until the copy has run)
        self.stream = self.stream_handle = None     # the stream that its last step was launched on


class RepeatedLayouts:
    """Which layouts have a captured step (``graphs``), the one used last at the end, and when the next one gets one: at the
    ``at``-th step of a layout, if there is a place among ``kept`` or a graph that has not been used for ``idle`` steps, which
    gives way.  The layout of a graph that gave way counts anew.  So there are ``kept`` captures in ``idle`` steps at most,
    whatever comes in whatever order, and layouts that come in turn keep the graphs that they have."""

    def __init__(self, at: int, kept: int, idle: int, counted: int):
        self.at, self.kept, self.idle, self.counted = at, kept, idle, counted
        self.graphs: dict = {}
        self.seen: dict = {}               # layout -> its steps up to the capture
        self._used: dict = {}              # the step that used a graph last
        self._steps = 0

    def replay(self, key):
        """The graph of a step's layout, or None (``to_capture`` is asked next then)."""
        graph = self.graphs.pop(key, None)
        if graph is not None:
            self._steps += 1
            self._used[key] = self._steps
            self.graphs[key] = graph
        return graph

    def to_capture(self, key) -> bool:
        """Count a step of a layout without a graph: is it the one to capture?  If so a graph that is in the way is dropped."""
        self._steps += 1
        seen = self.seen.get(key, 0) + 1
        if len(self.seen) > self.counted:
            self.seen.clear()
        self.seen[key] = seen
        if seen < self.at:
            return False
        if len(self.graphs) >= self.kept:
            oldest = next(iter(self.graphs))
            if self._steps - self._used[oldest] < self.idle:
                return False
            del self.graphs[oldest], self._used[oldest]
            self.seen.pop(oldest, None)
        return True

    def keep(self, key, graph) -> None:
        self._used[key] = self._steps
        self.graphs[key] = graph


class CapturedStep:
    def __init__(self, graph, logits, sampled, launches):
        self.graph, self.logits, self.sampled, self.launches = graph, logits, sampled, launches


class ModelRunner:
    """A model on one GPU with its cache.

    ``max_tokens``: tokens the cache pool holds; ``max_requests``: requests
    live at a time; ``page_size``: tokens per page (the reference's
    ``--block-size``, default 16, crates/vllm-scheduler/src/scheduler.rs:53).
    ``use_graphs``: steps in which every request brings exactly one token and
    wants its logits are replayed from a captured CUDA graph, other steps once
    their layout repeats (``RepeatedLayouts``)."""

    def __init__(self, model_dir, dtype="bfloat16", device="cuda:0", page_size: int = 16,
                 max_tokens: int = 16384, max_requests: int = 64, spec_override=None, use_graphs: bool = True):
        if not torch.cuda.is_available():
            raise RuntimeError("railgun_b200 runs on a CUDA device only; none is available")
        self.device = torch.device(device)
        torch.cuda.set_device(self.device)
        self.dtype = parse_dtype(dtype)
        # 32-bit means 32-bit: no reduced-precision matrix mode, no reduced-precision accumulation
        torch.backends.cuda.matmul.allow_tf32 = False
        torch.backends.cudnn.allow_tf32 = False
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
        self.arch, self.config, self.model = build_model(model_dir, self.dtype, self.device, spec_override)
        self.cache = CacheManager(self.model.cache_needs(), page_size, max_tokens, max_requests,
                                  self.dtype, self.device)
        self.views = _CacheViews(self.cache)
        self.page_sizes = [g.page_size for g in self.cache.groups]
        self.err_flag = torch.zeros(1, dtype=torch.int32, device=self.device)
        # graphs need every part to work from device-side descriptions only; a part that says it plans on the
        # host (none of the built-in ones) switches them off.  Per-request state is no obstacle: its buffers are
        # static and the rows' slots are data of the step (-1 in a padding row).
        self.use_graphs = bool(use_graphs) and self.model.graph_safe
        self._static: dict = {}
        # graph key -> ShapeGraph, of steps of ``shape_graph_min_tokens`` tokens and more and of shorter ones
        self._long_steps = RepeatedLayouts(2, SHAPE_GRAPHS_KEPT, GIVES_WAY_AFTER[0], LAYOUTS_COUNTED[0])
        self._short_steps = RepeatedLayouts(SMALL_GRAPH_AT, SMALL_GRAPHS_KEPT, GIVES_WAY_AFTER[1], LAYOUTS_COUNTED[1])
        self._shape_steps, self._shape_seen = self._long_steps.graphs, self._long_steps.seen
        self.shape_graph_min_tokens = SHAPE_GRAPH_MIN_TOKENS
        self._graph_pool = None
        self._ctx_hint = 0
        self.last_h2d_bytes = 0
        self.last_greedy = None
        self._greedy_host = None

    @property
    def alloc(self):
        return self.cache.alloc

    # ---- the step function -----------------------------------------------------------------------
    def step(self, entries) -> torch.Tensor | None:
        """Run one batch; float32 logits [wanted, vocab] in the order of the
        entries and of each entry's ``want``, or None if nothing is wanted.
        The result may be a view of a buffer the next step overwrites (of steps
        of single tokens, and of ``shape_graph_min_tokens`` tokens and more)."""
        entries = [e if isinstance(e, StepEntry) else StepEntry(*e) for e in entries]
        if NVTX:
            torch.cuda.nvtx.range_push(f"step {len(entries)} requests {sum(len(e.tokens) for e in entries)} tokens")
            try:
                return self._step(entries)
            finally:
                torch.cuda.nvtx.range_pop()
        return self._step(entries)

    def _step(self, entries):
        self.last_greedy = None
        if self.use_graphs and entries and all(
                len(e.tokens) == 1 and list(e.want) == [0] and self.alloc.has(e.request_id) for e in entries):
            return self._step_decode_graph(entries)
        if self.use_graphs and entries:
            return self._step_shape_graph(entries)
        batch = build_step_batch(entries, self.alloc, self.page_sizes, self.model.vocab_size,
                                 self.model.spec.max_position, self.device, self.err_flag)
        self.last_h2d_bytes = batch.h2d_bytes
        logits = self.model.forward(batch, self.views)
        self._commit(entries, batch)
        return logits

    def _in_order(self, owner) -> None:
        """The buffers of a captured step (``owner``) are its steps' one after the other: launched on another stream than the
        last time, a step waits for what is on that one."""
        handle = ops.current_stream_handle()
        if owner.stream_handle == handle:
            return
        stream = torch.cuda.current_stream(self.device)
        if owner.stream is not None:
            stream.wait_stream(owner.stream)
        owner.stream, owner.stream_handle = stream, handle

    def _commit(self, entries, batch) -> None:
        self.alloc.commit_many(batch.host_request_ids, batch.host_context_lens)

    def _step_shape_graph(self, entries):
        """Steps (portions of prompts) whose packed layout was seen before
        replay a CUDA graph captured for that layout: token counts, wanted places
        and block-table widths fix every shape, everything else is data in the
        step's one device buffer.  The first steps of a layout run eagerly, the
        second (of a short step the ``SMALL_GRAPH_AT``-th) is captured while it runs, later
        ones replay; a few layouts are kept (``RepeatedLayouts``)."""
        steps = (self._long_steps if sum(len(e.tokens) for e in entries) >= self.shape_graph_min_tokens
                 else self._short_steps)
        build = lambda into: build_step_batch(entries, self.alloc, self.page_sizes, self.model.vocab_size,
                                              self.model.spec.max_position, self.device, self.err_flag, into=into,
                                              splits=self.model.single_token_splits)

        result = None

        def known(key):
            nonlocal result
            shape = steps.graphs.get(key)
            if shape is None:
                return None
            self._in_order(shape)                                  # the step is copied into its buffer next
            # a short step's logits are the caller's, as they are where its kernels are launched one by one
            result = shape.logits if steps is self._long_steps or shape.logits is None else torch.empty_like(shape.logits)
            return shape.dev, (0 if result is shape.logits else result.data_ptr())

        batch = build(known)
        self.last_h2d_bytes = batch.h2d_bytes
        key = batch.graph_key
        shape = steps.replay(key)
        if shape is not None:
            # the step was packed straight into the graph's buffer: launch
            shape.hold = batch
            shape.graph.replay()
            ops.launch_counter().value += shape.launches
            ops.mark_tc_unchecked()
            self._commit(entries, batch)
            return result
        if not steps.to_capture(key):
            logits = self.model.forward(batch, self.views)
            self._commit(entries, batch)
            return logits
        # the layout repeats: a static copy of the packed buffer, one eager run over it (this step), the capture
        dev = torch.empty(batch.host_buffer.numel(), dtype=torch.int32, device=self.device)
        batch = build(lambda key: (dev, 0))
        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            eager = self.model.forward(batch, self.views)
            eager = eager.clone() if eager is not None else None
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        counter = ops.launch_counter()
        n0 = counter.value
        graph = torch.cuda.CUDAGraph()
        with capture(graph):
            logits = self.model.forward(batch, self.views)
            if steps is self._short_steps and logits is not None:
                logits = logits.contiguous()
                ops.step_result(logits, batch.result_address[-2:])
        launches = counter.value - n0
        counter.value = n0
        shape = ShapeGraph(dev, batch, graph, logits, launches)
        self._in_order(shape)
        steps.keep(key, shape)
        self._commit(entries, batch)
        return eager

    def end(self, request_ids) -> None:
        """The requests are finished: their pages and slots come back."""
        for rid in request_ids:
            if self.alloc.has(rid):
                self.alloc.release(rid)

    def check_device_errors(self) -> None:
        """Raise if a kernel gave up a bounded wait or met a position outside its table since the last check
        (synchronises).  Steps replayed from decode graphs carry their own flag, which also travels to the host
        with their tokens."""
        ops.tc_gemm_check()
        flags = [self.err_flag] + [st.out_dev[st.B:] for st in self._static.values()]
        code = int(torch.cat(flags).max().item())
        if code:
            for f in flags:
                f.zero_()
            raise_device_error(code)

    # ---- decode steps from captured graphs -----------------------------------------------------------
    def _static_for(self, n_requests: int, max_context: int) -> StaticDecodeBatch:
        """The static batch for so many requests whose longest context is this: of the narrowest tables that hold it."""
        B = _bucket(n_requests, _BATCH_BUCKETS)
        # block tables are as wide as the group with the smallest pages needs
        page = min(self.page_sizes) if self.page_sizes else 16
        ctx_bucket = SHORT_CONTEXT
        while -(-ctx_bucket // page) * page < max_context:
            ctx_bucket = max(1024, 2 * ctx_bucket)
        key = (B, -(-ctx_bucket // page))
        if key not in self._static:
            self._static[key] = StaticDecodeBatch(self, *key)
        return self._static[key]

    def _capture(self, static: StaticDecodeBatch, follow: FollowStep | None = None,
                 sampling: bool = False) -> CapturedStep:
        """Capture one decode step over the static buffers: the copy of its
        packed inputs from pinned memory, the forward pass, the choice of the
        tokens and their copy to pinned memory, so that one graph launch and one
        wait are all the host does.  With ``follow`` the step takes its token
        ids from the step before it on the device and everything else from
        ``follow``'s pinned buffer.  With ``sampling`` the tokens are drawn with
        the rows' parameters in the static buffer (temperature 0: greedy)
        instead of the plain argmax.

        The step whose arrival makes the capture necessary runs here, once,
        outside the capture (libraries set themselves up in that run); the
        graph serves the steps after it.  So a step is executed exactly once,
        which a part with state of its own needs (rewriting a cache entry is
        harmless, advancing a state twice is not).  Returns the captured step
        and that first run's logits."""
        counter = ops.launch_counter()
        B = static.B

        def body():
            if follow is not None:
                ops.step_in(follow.host_in, static.dev, first=B)
            else:
                ops.step_in(static.host, static.dev, seq=static.seq, done=static.blocks_done)
            # a following step reads its token ids where the step before left its greedy tokens
            batch = static.batch if follow is None else dataclasses.replace(static.batch, token_ids=static.sampled)
            logits = self.model.forward(batch, self.views)
            if sampling:
                sp = static.sampling
                sampled = ops.sample(logits, sp["temperature"], sp["top_k"], sp["top_p"], sp["seed"],
                                     sp["counter"], out=static.sampled)
            else:
                sampled = ops.argmax(logits, out=static.sampled)
            ops.step_out(static.out_dev, (follow or static).host_out)
            return logits, sampled

        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            first_logits, _ = body()                        # this step itself
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        n0 = counter.value
        with capture(graph):
            logits, sampled = body()
        launches = counter.value - n0
        counter.value = n0
        return CapturedStep(graph, logits, sampled, launches), first_logits

    def _step_decode_graph(self, entries) -> torch.Tensor:
        R = len(entries)
        ids = np.fromiter((e.request_id for e in entries), dtype=np.int64, count=R)
        tokens = np.fromiter((e.tokens[0] for e in entries), dtype=np.int32, count=R)
        if len(set(ids.tolist())) != R:
            raise BatchError("a request appears twice in one step")
        return self.decode_step_flat(ids, tokens)

    def decode_step_flat(self, ids: np.ndarray, tokens: np.ndarray) -> torch.Tensor:
        """One decode step for requests already in the cache: ``ids`` int64
        (distinct), ``tokens`` int32, one token each, logits wanted for all.
        Returns the logits [R, V] (a view of a static buffer); the tokens the
        graph chose are in ``last_greedy``: for a request whose slot record has
        a temperature above zero a draw with the record's parameters (numbered
        by its count of generated tokens), else the argmax."""
        R = len(ids)
        self.last_greedy = None
        if tokens.min() < 0 or tokens.max() >= self.model.vocab_size:
            raise BatchError(f"token ids must be in [0, {self.model.vocab_size})")
        longest = lambda: 1 + max((self.alloc.num_computed(i) for i in ids.tolist() if self.alloc.has(i)), default=0)  # noqa: E731
        # mostly the last step's requests, a token further on.  Where they are others the tables may turn out too narrow, or
        # wider than this step's own: what a step computes does not depend on the one before it, so it is packed anew
        ctx = self._ctx_hint + 1 if self._ctx_hint else longest()
        while True:
            static = self._static_for(R, ctx)
            static.wait_until_reusable()
            try:
                sampled = self.alloc.pack_decode(ids, static.B, static.MB, static.host_np[static.B:],
                                                 sampling=static.host_np[static.sampling_off:])
            except CacheError as e:
                if "bad argument" in str(e) and ctx < self.model.spec.max_position:
                    ctx = min(max(2 * ctx, longest()), self.model.spec.max_position)
                    continue
                raise
            B = static.B
            ctx = self._ctx_hint = int(static.host_np[2 * B:2 * B + R].max())
            if ctx > self.model.spec.max_position:
                raise BatchError(f"position {ctx - 1} is beyond the model's max_position_embeddings "
                                 f"{self.model.spec.max_position}")
            if self._static_for(R, ctx) is static:
                break
        static.host_np[:R] = tokens
        static.host_np[R:B] = 0
        static.packed()
        self.last_h2d_bytes = static.host.numel() * 4
        self._in_order(static)
        key = sampled
        logits = None
        if key not in static.step_graphs:
            static.step_graphs[key], logits = self._capture(static, sampling=key)   # runs this step and captures it
        cap = static.step_graphs[key]
        if logits is None:
            cap.graph.replay()                              # upload, the step, greedy tokens back to pinned memory
            ops.launch_counter().value += cap.launches
            logits = cap.logits
        if static.in_flight is None:
            static.in_flight = torch.cuda.Event()
        static.in_flight.record()
        self.alloc.advance(ids, 1)
        self.last_greedy = cap.sampled[:R]
        self._greedy_host = (static, R)
        return logits[:R]

    def greedy_tokens_host(self):
        """The tokens that the last graph-replayed decode step chose (its argmax,
        or its draws if it was given sampling parameters) as a numpy array; waits
        for the step, whose graph copied them to pinned memory itself.  None if
        the last step was not such a step."""
        if self.last_greedy is None or self._greedy_host is None:
            return None
        static, R = self._greedy_host
        static.in_flight.synchronize()
        static.raise_if_flagged(static.host_out_np)
        return static.host_out_np[:R].copy()

    def decode_follow(self, ids: np.ndarray, after) -> FollowStep | None:
        """Launch the decode step that follows a launched one for the same
        requests (``ids`` int64, in its row order) before that one's tokens are
        on the host: the token ids stay on the device.  ``after`` is what that
        step ran on: the FollowStep it was, or None for the step that
        ``decode_step_flat`` launched last.  Its draws are numbered one after
        those of that step.  Nothing is committed: the caller
        commits the step once it knows that the requests went on.  Returns None
        if the step cannot be launched this way (no pages, a context beyond the
        static batch's tables or the model's positions)."""
        if after is None:
            if self._greedy_host is None:
                return None
            static, R = self._greedy_host
            k = 0
        else:
            static, R = after.static, len(after.ids)
            k = 1 - static.follow.index(after)
        if R != len(ids):
            return None
        if static.follow[k] is None:
            static.follow[k] = FollowStep(static)
        f = static.follow[k]
        if not f.done.query():                              # only after a launch that was dropped: its copies may be pending
            f.done.synchronize()
        B = static.B
        ahead = 0 if after is None else 1                   # decode_step_flat has advanced its requests already
        try:
            key = self.alloc.pack_decode(ids, B, static.MB, f.host_in_np[B:], ahead=ahead,
                                         sampling=f.host_in_np[static.sampling_off:], draw_ahead=1)
        except CacheError:
            return None
        if int(f.host_in_np[2 * B:2 * B + R].max()) > self.model.spec.max_position:
            return None
        self._in_order(static)
        if key not in f.captured:
            f.captured[key], _ = self._capture(static, follow=f, sampling=key)       # runs this step and captures it
        else:
            f.captured[key].graph.replay()
            ops.launch_counter().value += f.captured[key].launches
        f.done.record()
        self.last_h2d_bytes = (static.host.numel() - B) * 4
        f.ids = ids.copy()
        return f
