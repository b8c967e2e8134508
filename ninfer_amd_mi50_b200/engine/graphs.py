"""Decode steps replayed from CUDA graphs.

A decode-only step launches a few hundred small kernels; issuing them from the host
costs more than running them.  The reference has an opt-in HIP-graph path for its
one-token forward, dense models only, because its MoE routing synchronises with the host
(src/models/model.hip:786-830; src/runtime/engine.cpp:151-154).  Here routing stays on the
device, so the whole step is captured: one graph per (number of rows, context bound).
A step copies its index data into the graph's fixed input buffer and replays it.

Rows beyond the live requests are padding: token 0 at position 0 of a request whose only
page is the cache's null page.  They cost a little work and touch nothing that is read.
"""

from __future__ import annotations

import gc
from typing import Dict, List, Optional, Sequence, Tuple

import numpy as np
import torch

from ..kernels import lib as klib
from ..parts.base import StepContext
from .batch import StepEntry


def row_bucket(n: int) -> int:
    """Rows a graph is built for: exact up to 8, then the next power of two."""
    if n <= 8:
        return n
    b = 16
    while b < n:
        b <<= 1
    return b


def context_bucket(n: int, limit: int) -> int:
    """Context bound a graph is built for: the next multiple of 512 (the decode attention
    launches one block of CTAs per 128 keys of this bound, so a tight bound saves idle CTAs)."""
    return min((n + 511) // 512 * 512, max(limit, 1))


STAGES = 16                          # steps whose index data may be on its way, at most ...
STAGING_BYTES = 32 << 20             # ... and what the buffers of all of them may take, two kept in any case


class Staging:
    """Pinned buffers out of which a runner's graphs send their steps' index data, used in turn, each with the event of its
    last copy: the host runs ahead of the device on purpose, so the copy out of a buffer may still be queued when the next
    steps are being prepared; a buffer is rewritten only after its own last copy has finished.  They belong to no graph:
    each is filled from end to end at every step, and there are no more of them for a service that has passed through many
    row counts and context bounds.  As many as STAGES steps ahead is what a caller gets that knows its tokens beforehand:
    the time that decode steps give the host is what it prepares the next prompt's eager step in (with two buffers it waited
    a step's length at every step: 1.4 of 5.3 ms over four prompts of 2,048 tokens and 12 decode steps).  Generation, which
    reads every step's tokens, is one step ahead."""

    def __init__(self):
        self.hosts: List[torch.Tensor] = []
        self.nps: List[np.ndarray] = []
        self.views: Dict[int, List[torch.Tensor]] = {}          # their first so many numbers, one entry a row count
        self.copied: List[Optional[torch.cuda.Event]] = []      # made at the first use, recorded again at every other
        self.turn = 0

    def fit(self, total: int) -> None:
        """Buffers of `total` int32 numbers at least, and their views of that many."""
        if self.hosts and self.hosts[0].numel() >= total:
            self.views.setdefault(total, [h[:total] for h in self.hosts])
            return
        for e in self.copied:
            if e is not None:
                e.synchronize()
        stages = max(2, min(STAGES, STAGING_BYTES // (4 * total)))
        self.hosts = list(torch.empty((stages, total), dtype=torch.int32).pin_memory().unbind(0))
        self.nps = [h.numpy() for h in self.hosts]
        self.views = {n: [h[:n] for h in self.hosts] for n in [*self.views, total]}
        self.copied, self.turn = [None] * stages, 0

    def take(self) -> int:
        """The buffer to fill next; waits for the copy that last read it."""
        i = self.turn % len(self.hosts)
        self.turn += 1
        if self.copied[i] is not None:
            self.copied[i].synchronize()
        return i

    def send(self, i: int, dev: torch.Tensor) -> None:
        dev.copy_(self.views[dev.numel()][i], non_blocking=True)
        if self.copied[i] is None:
            self.copied[i] = torch.cuda.Event()
        self.copied[i].record(torch.cuda.current_stream(dev.device))


class DecodeGraph:
    def __init__(self, runner, staging: Staging, rows: int, context_bound: int):
        self.runner, self.staging, self.S, self.context_bound = runner, staging, rows, context_bound
        cache, dev = runner.cache, runner.device
        S = rows
        self.width = cache.max_pages_per_request
        sizes = [S, S, S, S + 1, S, S, S] + [S * self.width for _ in cache.groups]
        self.offsets = np.cumsum([0] + sizes).tolist()
        total = self.offsets[-1]
        self.dev = torch.zeros((total,), dtype=torch.int32, device=dev)
        parts = [self.dev[self.offsets[i]:self.offsets[i + 1]] for i in range(len(sizes))]
        self.ctx = StepContext(
            dtype=runner.dtype, device=dev, T=S, S=S, token_ids=parts[0], positions=parts[1],
            row_seg=parts[2], seg_row0=parts[3], seg_pos0=parts[4], seg_slot=parts[5],
            logit_rows=parts[6], seg_len_host=[1] * S, seg_pos0_host=None, max_rows_per_seg=1,
            max_context=context_bound, graph_mode=True)
        for gi, g in enumerate(cache.groups):
            self.ctx.block_tables[g.index] = parts[7 + gi].view(S, self.width)
        # a row is its own segment, and its logits are wanted: row_seg, seg_row0 and logit_rows of every step
        self.counting = np.concatenate([np.arange(S), np.arange(S + 1)]).astype(np.int32)
        staging.fit(total)
        i = staging.take()
        self._fill(staging.nps[i], [], [])
        staging.send(i, self.dev)
        # warm up on a side stream (library handles, lazily set kernel attributes), then capture
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            for _ in range(2):
                runner.run(self.ctx)
        torch.cuda.current_stream(dev).wait_stream(side)
        torch.cuda.synchronize(dev)
        before = klib.launch_count()
        self.graph = torch.cuda.CUDAGraph()
        # No cyclic garbage collection while the stream captures: collecting an older engine's
        # graphs then would destroy them inside this capture, which the runtime forbids and
        # answers by invalidating the capture.
        collecting = gc.isenabled()
        gc.collect()
        gc.disable()
        try:
            with torch.cuda.graph(self.graph):
                self.logits = runner.run(self.ctx)
        finally:
            if collecting:
                gc.enable()
        self.kernels = klib.launch_count() - before
        self.h2d_bytes = total * 4

    def _fill(self, a: np.ndarray, entries: Sequence[StepEntry], lengths: Sequence[int]) -> None:
        cache, o, S = self.runner.cache, self.offsets, self.S
        n = len(entries)
        a[o[0]:o[0] + n] = [int(e.tokens[0]) for e in entries]
        a[o[0] + n:o[1]] = 0
        a[o[1]:o[1] + n] = lengths
        a[o[1] + n:o[2]] = 0
        a[o[2]:o[4]] = self.counting
        a[o[6]:o[7]] = self.counting[:S]
        a[o[4]:o[4] + n] = lengths
        a[o[4] + n:o[5]] = 0
        slots = [cache.slot(e.req) for e in entries]
        a[o[5]:o[5] + n] = slots
        a[o[5] + n:o[6]] = cache.null_slot
        for gi, g in enumerate(cache.groups):
            tbl = a[o[7 + gi]:o[8 + gi]].reshape(S, self.width)
            if n:
                tbl[:n] = cache.block_rows(g.index, slots, self.width)
            tbl[n:, 0] = g.null_page
            tbl[n:, 1:] = -1

    def run(self, entries: Sequence[StepEntry], device_tokens: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Pages for the new tokens are reserved already.  Returns logits [S, vocab] that stay
        valid until the next replay of this graph.  `device_tokens` (int32 [len(entries)] on the
        device) replace the entries' token ids: the tokens a step before has just drawn, which
        the host has not read yet."""
        lengths = [self.runner.cache.length(e.req) for e in entries]
        i = self.staging.take()
        self._fill(self.staging.nps[i], entries, lengths)
        self.staging.send(i, self.dev)
        if device_tokens is not None:
            self.dev[self.offsets[0]:self.offsets[0] + len(entries)].copy_(device_tokens)
        self.graph.replay()
        klib.count_launches(self.kernels)
        return self.logits


class DecodeGraphs:
    """The runner's graphs, built on first use."""

    def __init__(self, runner, max_rows: int):
        self.runner, self.max_rows = runner, max_rows
        self.staging = Staging()
        self.graphs: Dict[Tuple[int, int], DecodeGraph] = {}

    def eligible(self, entries: Sequence[StepEntry]) -> bool:
        return 0 < len(entries) <= self.max_rows and all(len(e.tokens) == 1 for e in entries)

    def get(self, entries: Sequence[StepEntry]) -> DecodeGraph:
        cache = self.runner.cache
        rows = row_bucket(len(entries))
        longest = max(cache.length(e.req) for e in entries) + 1
        key = (rows, context_bucket(longest, cache.max_context))
        if key not in self.graphs:
            self.graphs[key] = DecodeGraph(self.runner, self.staging, *key)
        return self.graphs[key]
