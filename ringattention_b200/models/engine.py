"""The serving loop shared by the inference engines: chunked prefill, decoding one token per sequence and step (eagerly or
as one replayed CUDA graph), greedy sampling, and the step counters on the device that make a decode step replayable.

An engine supplies ``prefill_chunk`` (append a chunk, return the last position's logits), ``_decode_body`` (all launches of
one decode step, every per-token scalar read from ``state``) and ``_clear_cache``."""
from __future__ import annotations

import time
from typing import List

import torch

from ..ops import kernels as K

# Free memory of the device below which the allocator gives its cached blocks back before a step is recorded. While a capture is under way it
# cannot, and the private pool of a capture takes none of them: the recording would run out of memory beside gigabytes of cached blocks, or
# leave the driver nothing to upload the graph with. A step's own buffers are megabytes (the partial results of 512 splits of 64 heads 17, the
# logits of eight sequences 1.5); the first capture of a process took 72 from the driver.
RECORD_ROOM = 1 << 30


class InferenceEngine:
    def __init__(self, batch: int, device, token_rows: int):
        self.device = torch.device(device)
        self.B = batch
        self.length = 0                             # tokens in the cache (global)
        # [position, step] on the device: lets one recorded CUDA graph serve every decode step
        self.state = torch.zeros(2, dtype=torch.int64, device=self.device)
        self._graph = None
        self._old_graph = None                      # one that no longer serves: the next one takes over its buffers
        self._recorded = None                       # launch constants of the recorded step
        self._reset_since = False                   # reset() since it was recorded or found to serve
        self._state_at = 0                          # position in `state`
        self._tok_buf = torch.zeros(token_rows, dtype=torch.int32, device=self.device)

    # ------------------------------------------------------------------ supplied by the engine
    def prefill_chunk(self, tokens: torch.Tensor) -> torch.Tensor:
        raise NotImplementedError

    def _decode_body(self, tokens: torch.Tensor) -> torch.Tensor:
        raise NotImplementedError

    def _clear_cache(self) -> None:
        raise NotImplementedError

    def _check_room(self, n: int) -> None:
        """Raise when ``n`` more tokens do not fit (engines with a fixed cache size override it)."""

    def first_tokens(self, logits: torch.Tensor) -> torch.Tensor:
        """The tokens decoding starts with, from the prompt's last logits."""
        return self.sample(logits)

    # ------------------------------------------------------------------ sampling
    @staticmethod
    def sample(logits: torch.Tensor) -> torch.Tensor:
        """Greedy."""
        return logits.argmax(dim=-1)

    # ------------------------------------------------------------------ decode
    def _set_position(self) -> None:
        self.state[0] = self._state_at = self.length

    @torch.no_grad()
    def decode_step(self, tokens: torch.Tensor) -> torch.Tensor:
        """One token per sequence: ``tokens (B,)`` -> logits ``(B, vocab)`` fp32 (same on all ranks)."""
        self._check_room(1)
        self._set_position()
        logits = self._decode_body(tokens.to(self.device, torch.int32).reshape(-1).contiguous())
        self.length += 1
        self._state_at = self.length
        return logits

    @torch.no_grad()
    def decode_step_graph(self) -> torch.Tensor:
        """Greedy step on the token in ``self._tok_buf`` through a CUDA graph recorded on first use (see :meth:`launch_constants`):
        one replay per token instead of a handful of launches per layer. Writes the next token back into
        ``self._tok_buf`` and returns it. Call :meth:`decode_step` at least once before (buffers and
        kernels must exist before capture)."""
        self._check_room(1)
        if self._state_at != self.length:
            self._set_position()
        if not self._graph_serves():
            self._graph, self._old_graph = None, self._graph or self._old_graph
            self._graph = self._record(self._greedy_step)
            self._recorded = self._constants()
        self._reset_since = False
        self._graph.replay()
        self.length += 1
        self._state_at = self.length
        return self._tok_buf

    def launch_constants(self):
        """Everything that a recorded decode step holds and that may be another thing for the next prompt, as plain values that compare by
        ``==`` (addresses and layouts of the weights and caches, the configuration): after a :meth:`reset` the step is replayed if these are
        still the same. None: record again after every reset (the default; also for a step with addresses in it that others
        may free, as of buffers that are shared with peers or with other engines)."""
        return None

    def _constants(self):
        # a sampler of the caller's own may hold anything
        return self.launch_constants() if self.sample is InferenceEngine.sample else None

    def _graph_serves(self) -> bool:
        if self._graph is None or not self._reset_since:
            return self._graph is not None
        now = self._constants()
        return now is not None and now == self._recorded

    def _greedy_step(self) -> None:
        logits = self._decode_body(self._tok_buf)
        if self.sample is InferenceEngine.sample and logits.is_cuda and logits.dtype == torch.float32 and logits.stride(-1) == 1:
            K.greedy(logits, self._tok_buf)  # what sample() and the cast say, in one launch
        else:
            self._tok_buf.copy_(self.sample(logits).to(torch.int32))

    def _record(self, body) -> torch.cuda.CUDAGraph:
        """Record ``body`` as ``torch.cuda.graph`` does, but leave the allocator's cached blocks alone while the device has room
        (:data:`RECORD_ROOM`): emptying the cache before every prompt's recording made the next prompt's prefill allocate all of
        its buffers from the driver again. A step that needs more than there was is recorded again without the cache. The buffers of
        the graph recorded before are taken over (it is dropped here)."""
        # Eager steps sample without this kernel: it would be loaded while the capture is under way. The first one of a process took 19 to 76 ms so, on
        # two machines; 19 to 20 with the kernel there.
        if self.sample is InferenceEngine.sample and self.device.type == "cuda":
            K.greedy(torch.zeros(1, 1, device=self.device), torch.empty(1, device=self.device, dtype=torch.int32))
        torch.cuda.synchronize()
        low = torch.cuda.mem_get_info(self.device)[0] < RECORD_ROOM
        for again in (False, True):
            if low or again:
                torch.cuda.empty_cache()
            try:
                graph = self._capture(body)
                break
            except torch.OutOfMemoryError:
                if again:
                    raise
        self._old_graph = None
        return graph

    def _capture(self, body) -> torch.cuda.CUDAGraph:
        g = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream(self.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            if self._old_graph is None:
                g.capture_begin()
            else:
                g.capture_begin(pool=self._old_graph.pool())
            try:
                body()
            finally:
                g.capture_end()
        torch.cuda.current_stream().wait_stream(side)
        return g

    def reset(self) -> None:
        """Forget the cached context (the cache memory is kept). The recorded decode graph stays if its launch constants do."""
        self.length = 0
        self.state.zero_()
        self._state_at = 0
        self._reset_since = True
        self._clear_cache()

    # ------------------------------------------------------------------ generation
    @torch.no_grad()
    def generate(self, prompt: torch.Tensor, new_tokens: int, chunk: int = 32768, use_graph: bool = True):
        """Chunked prefill of ``prompt (B, T)`` followed by greedy decoding. Returns the generated
        tokens ``(B, new_tokens)`` and timing: prefill seconds, per-token decode latencies."""
        B, T = prompt.shape
        if self.length:
            self.reset()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        logits = None
        for c0 in range(0, T, chunk):
            logits = self.prefill_chunk(prompt[:, c0:c0 + chunk])
        torch.cuda.synchronize()
        t_prefill = time.perf_counter() - t0
        out: List[torch.Tensor] = []
        marks: List[tuple] = []
        nxt = self.first_tokens(logits)
        eager = 0 if self._graph_serves() else 2    # buffers and kernels must exist before a step is recorded
        for i in range(new_tokens):
            out.append(nxt.clone())
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            if use_graph and i >= eager:
                if i == eager:
                    self._tok_buf.copy_(nxt.to(torch.int32))
                nxt = self.decode_step_graph()
            else:
                nxt = self.sample(self.decode_step(nxt))
            e1.record()
            marks.append((e0, e1))
        # The host waits once, not for every token: between two steps the device otherwise idles for as long as the host takes to wake up
        # and launch the next one.
        torch.cuda.synchronize()
        return (torch.stack([t.to(torch.int64) for t in out], dim=1),
                {"prefill_s": t_prefill, "decode_ms": [a.elapsed_time(b) for a, b in marks]})
