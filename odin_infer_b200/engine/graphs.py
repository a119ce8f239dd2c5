"""CUDA graphs of the decode step.

A step in which every sequence brings one token launches a few hundred small
kernels; at small batches the launches cost more than the kernels.  Such steps
are captured once per batch-size bucket and replayed: the step's integer tables
live in fixed device buffers that are refilled before every replay, padding rows
(sequence -1) make up the difference to the bucket size and change no result.

Only a model whose parts all say `graph_safe` is captured (the engine asks before it
builds this object).  A step that finds no graph yet runs eagerly, and that run IS the
step: the capture that follows records the same launches for later steps without
executing them, so nothing (keys, values, a mixer's fixed-size state) is applied twice.

In 32-bit the capture waits until a shape of step comes for the second time.  A capture costs as much as several
eager steps, and 32-bit engines often see each shape once: a port of weights is checked with a few prompts of
different lengths.

Engines in several threads do not disturb one another's captures: each records on a stream of its own, in
the mode in which other threads may allocate, and nothing here waits for the whole device or gives the
allocator's cache back, as `torch.cuda.graph` does on its way in (a wait for the device ends any capture under
way).  The same holds for what the caller's other threads do: `torch.cuda.synchronize()` in one of them
ends a capture with an error; waiting for a stream or an event does not.
"""
from __future__ import annotations

import torch

from ..csrc import ops
from .step import StepBatch, StepEntry

BUCKETS = (1, 2, 4, 8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256)

# Short prompts are launch-bound too when they run eagerly (a few hundred launches of ~25 us of host
# time each: 8 ms for what the device does in 3): steps of a few sequences with up to 1,024 tokens in
# all are captured as well, per bucket of their token count and of their number of sequences, padded
# with rows of sequence -1 and with empty sequences.  16 rows: the products then take tiles of 16 tokens and cut K
# otherwise than at 32, so bfloat16 logits of prompts of up to 16 tokens differ from those of a bucket of 32 by rounding.  9
# tokens on the 1.7B size: 1.31 ms (1.57 padded to 32), on the 8B size 3.19 (3.54), on eight layers of recurrences 0.76 (1.07),
# on eight with experts 1.05 (1.03).
PROMPT_BUCKETS = (16, 32, 64, 128, 192, 256, 384, 512, 768, 1024)
PROMPT_SEQ_BUCKETS = (1, 2, 4, 8, 16)

# In 32-bit only up to 256 tokens, and at most one wanted place per sequence: beyond that a step of a model that is not
# tiny keeps the device busy for longer than its launches take (the 1.7B size: the products of 64 rows alone 9.3 ms beside
# 5.8 ms of launches), while the padding rows cost their share of it; up to there the buckets from 64 on are multiples of the
# products' 64-row tiles.
PROMPT_ROWS_32BIT = 256


def bucket_for(n: int) -> int | None:
    for b in BUCKETS:
        if n <= b:
            return b
    return None


class DecodeGraphs:
    def __init__(self, rt, model, cache):
        self.rt, self.model, self.cache = rt, model, cache
        self._graphs: dict[tuple, tuple] = {}
        # In 32-bit a step keeps the forms that its own lengths choose, whatever the bucket and whoever shares it, so that its
        # bits are those of the eager step; in bfloat16 the bucket's rows choose.
        self._exact_forms = rt.dtype == torch.float32
        self._forms_from = model.forms_from if self._exact_forms else ()
        self._short_contexts: dict[int, int] = {}   # bucket -> DecoderModel.short_context
        self._seen: set[tuple] = set()   # 32-bit: keys of steps that came once and ran eagerly
        # In 32-bit, whose logits are copied out right behind a replay, the graphs share their scratch memory: they replay one
        # after the other on one stream, and nothing of a replay but its logits is read after it.
        self._pool = torch.cuda.graph_pool_handle() if rt.dtype == torch.float32 else None
        self._stream = None              # the captures' own, made at the first of them
        self.last_h2d_bytes = 0

    def takes(self, entries: list[StepEntry]) -> bool:
        """Is this a step that `run` may replay a graph for?"""
        if all(len(e.tokens) == 1 for e in entries):
            return True
        if self.rt.dtype == torch.float32 and (sum(len(e.tokens) for e in entries) > PROMPT_ROWS_32BIT
                                               or any(len(e.want) > 1 for e in entries)):
            return False
        return (len(entries) <= PROMPT_SEQ_BUCKETS[-1] and sum(len(e.tokens) for e in entries) <= PROMPT_BUCKETS[-1]
                and any(e.want for e in entries))

    def _not_yet(self, key) -> bool:
        """Shall a step without a graph run eagerly and not be captured?"""
        if self.rt.dtype != torch.float32 or key in self._seen:
            return False
        self._seen.add(key)
        return True

    def _run_prompt(self, entries: list[StepEntry], starts: list[int]) -> torch.Tensor | None:
        """A few sequences' tokens (prompts or pieces of them) in a bucket of rows and of sequences."""
        n = sum(len(e.tokens) for e in entries)
        rows = next(b for b in PROMPT_BUCKETS if n <= b)
        seqs = next(b for b in PROMPT_SEQ_BUCKETS if len(entries) <= b)
        form = 0   # on which side of the lines between the parts' forms
        if self._forms_from:
            longest = max(len(e.tokens) for e in entries)
            form = sum(longest >= line for line in self._forms_from)
        key = ("prompt", rows, seqs, sum(len(e.want) for e in entries), form)
        hit = self._graphs.get(key)
        if hit is None:
            if self._not_yet(key):
                return NotImplemented
            batch = StepBatch(self.cache, entries, starts, self.rt.device, pad_rows_to=rows, pad_seqs_to=seqs,
                              exact_forms=self._exact_forms)
            return self._first_run(key, batch)
        graph, batch, logits, n_kernels = hit
        batch.fill(entries, starts)
        graph.replay()
        ops.add_launches(n_kernels)
        self.last_h2d_bytes = batch.h2d_bytes
        return self._handed_out(logits)

    def _handed_out(self, logits: torch.Tensor) -> torch.Tensor:
        """What a replay's caller gets: the graph's own buffer, which the next replay writes again; in 32-bit, whose logits
        are compared and kept, a copy."""
        return logits.clone() if self.rt.dtype == torch.float32 else logits

    def _first_run(self, key, batch: StepBatch, device_tokens=None) -> torch.Tensor | None:
        """The step itself, eagerly (first-use set-up of the kernels - function attributes, tensor
        maps, error flags, the allocator's pools - must not fall into a capture), then the capture
        of the same launches for the steps to come.  Returns the eager run's logits."""
        if device_tokens is not None:
            batch.take_tokens(*device_tokens)
        logits = self.rt.run(self.model, batch)
        torch.cuda.current_stream().synchronize()
        n0 = ops.launch_count()
        try:
            graph, captured = self._capture(batch)
        except torch.cuda.OutOfMemoryError:
            ops.add_launches(n0 - ops.launch_count())
            torch.cuda.empty_cache()          # the eager run's scratch memory, which the capture needs anew in its own pool
            graph, captured = self._capture(batch)
        n_kernels = ops.launch_count() - n0
        ops.add_launches(-n_kernels)          # recorded, not launched
        self._graphs[key] = (graph, batch, captured, n_kernels)
        self.last_h2d_bytes = batch.h2d_bytes
        return logits

    def _capture(self, batch: StepBatch) -> tuple:
        if self._stream is None:
            self._stream = torch.cuda.Stream(self.rt.device)
        graph = torch.cuda.CUDAGraph()
        try:
            with torch.cuda.stream(self._stream):
                graph.capture_begin(pool=self._pool, capture_error_mode="thread_local")
                try:
                    captured = self.rt.run(self.model, batch)
                finally:
                    graph.capture_end()
        except Exception:
            self._fresh_pool()
            raise
        return graph, captured

    def _fresh_pool(self) -> None:
        """A pool that no graph holds any more cannot be used again."""
        if self._pool is not None and not self._graphs:
            self._pool = torch.cuda.graph_pool_handle()

    def run(self, entries: list[StepEntry], starts: list[int], device_tokens=None) -> torch.Tensor | None:
        """Logits [wanted, vocab] of a one-token-per-sequence step (or of one sequence's short
        prompt), or NotImplemented if the batch is larger than the largest bucket or a 32-bit step
        of its shape came for the first time: such a step runs eagerly."""
        if any(len(e.tokens) > 1 for e in entries):
            return self._run_prompt(entries, starts)
        bucket = bucket_for(len(entries))
        if bucket is None:
            return NotImplemented
        # kernels whose launch shape follows the longest context (decode attention's key splits)
        # make a graph valid for a class of context lengths only: the class is part of the key
        longest = max(s + 1 for s in starts)
        short = self._short_contexts.get(bucket)
        if short is None:
            short = self._short_contexts[bucket] = self.model.short_context(self.rt, bucket)
        bucket = (bucket, "short" if longest <= short else self.rt.context_class(longest))
        hit = self._graphs.get(bucket)
        if hit is None:
            if self._not_yet(bucket):
                return NotImplemented
            batch = StepBatch(self.cache, entries, starts, self.rt.device, pad_rows_to=bucket[0], pad_seqs_to=bucket[0],
                              all_rows_wanted=True)
            logits = self._first_run(bucket, batch, device_tokens)
        else:
            graph, batch, logits, n_kernels = hit
            batch.fill(entries, starts)
            if device_tokens is not None:  # the tokens come from the device: into the tables after their copy
                batch.take_tokens(*device_tokens)
            graph.replay()
            ops.add_launches(n_kernels)
            self.last_h2d_bytes = batch.h2d_bytes
        rows = batch.wanted_rows
        if not rows:
            return None
        if rows == list(range(len(rows))):
            return logits[:len(rows)] if hit is None else self._handed_out(logits[:len(rows)])
        return logits[torch.tensor(rows, device=logits.device)]

    def clear(self) -> None:
        self._graphs.clear()
        self._seen.clear()
        self._fresh_pool()
