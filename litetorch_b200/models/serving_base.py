"""The part of cached serving that does not depend on the model: prompt chunks and batched decode steps over a paged cache
(and, for models with recurrent layers, per-sequence state slots), CUDA-graph replay of the decode step, sampling, and
`generate`.

A model supplies four pieces of device work and inherits the rest:

    _prompt_hidden(tokens, start, block_ids, slot)  hidden rows of a prompt chunk; writes the cache and the state
    _decode_hidden(d, S, width)                     hidden rows of one token of S sequences, from the packed input block
    _logits(hidden, rows)                           logits of the given rows (None: all)
    new_serving(...)                                on the engine: how to make the serving model (see `models.registry`)

The packed int32 input block of a decode step is [5 + width, S]: token, position, cache slot, context length, state slot
of every sequence, then its block table (transposed).

Inputs reach the device through pinned memory (the host allocator hands a block out again only when the copies out of it are
done), so that the host prepares a pass while the one before it runs: a copy from pageable memory, or a copy that is waited
for, ends when everything before it has run.
"""
from __future__ import annotations

import gc
from operator import index
from typing import List, Optional, Sequence

import numpy as np
import torch


def _ints(values: Sequence[int], n: int, dtype=np.int32) -> np.ndarray:
    """n whole numbers as an array.  They may be a tensor, or tensors of one element, on the device too (what a step returns)."""
    if isinstance(values, torch.Tensor):
        values = values.tolist()
    elif n and isinstance(values[0], torch.Tensor):
        values = map(int, values)
    return np.fromiter(values, dtype, n)


class ServingModel:
    state_slots = 0                          # > 0: the scheduler passes every sequence's state slot along

    def __init__(self, engine, block_size: int, graphs: bool):
        self.e = engine
        self.block_size = block_size
        self.graphs = graphs                 # record the decode step per (batch size, table width) and replay it
        self._graphs = {}
        self.sampler = None                  # None: greedy on the device; else a callable logits [rows, vocab] -> tokens
        self.last_logits = None              # [rows, vocab] of the newest step (kept for inspection and tests)
        self.prefill_tokens_computed = 0
        self.prefill_tokens_reused = 0

    # ------------------------------------------------------------------ the model's part
    def _prompt_hidden(self, tokens: Sequence[int], start: int, block_ids: Sequence[int], slot: int):
        raise NotImplementedError

    def _decode_hidden(self, d: torch.Tensor, S: int, width: int):
        raise NotImplementedError

    def _logits(self, hidden, rows: Optional[List[int]] = None) -> torch.Tensor:
        raise NotImplementedError

    def _warm_input(self, host: torch.Tensor) -> torch.Tensor:
        """The input block of the pass that runs a step before it is recorded; a model whose step changes more than the
        cache cells that the replay writes again points it at scratch."""
        return host

    # ------------------------------------------------------------------ tokens from logits
    def _pick(self, logits: torch.Tensor) -> torch.Tensor:
        self.last_logits = logits
        if self.sampler is not None:
            return self.sampler(logits.float())
        return self.e.K.argmax_rows(logits)

    # ------------------------------------------------------------------ prompt chunks
    @torch.no_grad()
    def prefill_chunk(self, tokens: Sequence[int], start: int, block_ids: Sequence[int], want_token: bool, slot: int = 0) -> int:
        """Run prompt positions [start, start + len(tokens)) of one sequence.  Returns the next token when `want_token` (the
        chunk completes the prompt), else -1."""
        self.prefill_tokens_computed += len(tokens)
        x = self._prompt_hidden(tokens, start, block_ids, slot)
        if not want_token:
            return -1
        return int(self._pick(self._logits(x, self._places([-1], len(tokens)))).item())

    @torch.no_grad()
    def score_chunk(self, tokens: Sequence[int], start: int, block_ids: Sequence[int], rows: Sequence[int], slot: int = 0) -> torch.Tensor:
        """The same pass; returns the fp32 logits [len(rows), vocab] at the given places among `tokens` (negative ones count from the end)."""
        self.prefill_tokens_computed += len(tokens)
        x = self._prompt_hidden(tokens, start, block_ids, slot)
        return self._logits(x, self._places(rows, len(tokens))).float()

    # ------------------------------------------------------------------ one token for every running sequence
    def _decode_body(self, d: torch.Tensor, S: int, width: int):
        logits = self._logits(self._decode_hidden(d, S, width))
        return logits, self._pick(logits)

    def _run_decode(self, last_tokens, positions, block_tables, slots):
        """(logits [S, vocab], next tokens [S]).  On a GPU the step's launches are recorded once per (batch size,
        block-table width) into a CUDA graph and replayed: the step then costs its kernels, not their launch overhead.  The
        inputs of a replay are copied into the graph's static input block first."""
        dev = self.e.device
        S = len(last_tokens)
        bs = self.block_size
        positions = [int(p) for p in positions]
        width = max((p + bs) // bs for p in positions)
        use_graph = self.graphs and dev.type == "cuda"
        if use_graph:
            width = (width + 15) // 16 * 16                     # fewer distinct graphs: table widths in steps of 16 blocks
        host = self._host(5 + width, S)
        h = host.numpy()
        h[0] = self._tokens(last_tokens, S)
        h[1] = positions
        h[2] = [int(t[p // bs]) * bs + p % bs for t, p in zip(block_tables, positions)]
        h[3] = h[1] + 1
        h[4] = 0 if slots is None else _ints(slots, S)
        n = [min(len(t), width) for t in block_tables]
        flat = np.concatenate([_ints(t if len(t) <= width else t[:width], k) for t, k in zip(block_tables, n)])
        table = np.zeros((S, width), np.int32)
        table[np.arange(width) < np.array(n)[:, None]] = flat
        h[5:] = table.T
        if not use_graph:
            return self._decode_body(host.to(dev, non_blocking=True), S, width)
        entry = self._graphs.get((S, width))
        if entry is None:
            static_in = self._warm_input(host).to(dev)
            side = torch.cuda.Stream(device=dev)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):                        # eager run on the capture stream: workspaces, caches
                self._decode_body(static_in, S, width)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            g, static_out = self._record(static_in, S, width, side)
            entry = self._graphs[S, width] = (g, static_in, static_out)
            # the eager pass wrote this step's cache cells already; the replay below rewrites the same ones
        g, static_in, static_out = entry
        static_in.copy_(host, non_blocking=True)
        g.replay()
        self.last_logits = static_out[0]
        return static_out

    def _record(self, static_in: torch.Tensor, S: int, width: int, side: torch.cuda.Stream):
        """(graph, outputs) of a decode step, recorded on `side`.  `torch.cuda.graph` gives all cached memory back first, which takes a tenth of a second
        and more after large states; here that is done where the device has less than 1 GB left (the driver keeps the graph there), and where the
        recording finds no memory: what lies free in the cache of another stream, or of the common pool, cannot be used, nor given back, while it is
        under way."""
        for give_back in (torch.cuda.mem_get_info(side.device)[0] < 1 << 30, True):
            if give_back:
                torch.cuda.synchronize()
                gc.collect()
                torch.cuda.empty_cache()
            g, short = torch.cuda.CUDAGraph(), None
            with torch.cuda.stream(side):
                g.capture_begin()
                try:
                    out = self._decode_body(static_in, S, width)
                except torch.cuda.OutOfMemoryError as e:
                    short = e.with_traceback(None)             # (its frames hold what was made so far)
                finally:
                    g.capture_end()
            if short is None:
                return g, out
            g.reset()
        raise short

    @torch.no_grad()
    def decode_batch(self, last_tokens: Sequence[int], positions: Sequence[int], block_tables: List[Sequence[int]],
                     slots: Optional[Sequence[int]] = None) -> List[int]:
        """last_tokens[s] sits at position positions[s] of sequence s and is not in the cache yet: run it and return the next
        token of every sequence."""
        return self._run_decode(last_tokens, positions, block_tables, slots)[1].tolist()

    @torch.no_grad()
    def decode_logits(self, last_tokens: Sequence[int], positions: Sequence[int], block_tables: List[Sequence[int]],
                      slots: Optional[Sequence[int]] = None) -> torch.Tensor:
        """The same step; returns its fp32 logits [S, vocab]."""
        out = self._run_decode(last_tokens, positions, block_tables, slots)[0]
        return out.clone() if out.dtype == torch.float32 else out.float()

    # ------------------------------------------------------------------ helpers
    def _host(self, *shape: int) -> torch.Tensor:
        """Host memory for 32-bit inputs, pinned where there is a GPU."""
        return torch.empty(shape, dtype=torch.int32, pin_memory=self.e.device.type == "cuda")

    def _tokens(self, tokens: Sequence[int], n: int) -> np.ndarray:
        return _ints(tokens, n)

    def _prompt_inputs(self, tokens: Sequence[int], start: int, block_ids: Sequence[int]):
        """(tokens, positions, cache slots, block table) of a portion on the device, int32, through one copy."""
        n, bs = len(tokens), self.block_size
        nb = (start + n + bs - 1) // bs
        host = self._host(3 * n + nb)
        h = host.numpy()
        p = np.arange(start, start + n, dtype=np.int32)
        table = _ints(block_ids[:nb], nb)
        h[:n] = self._tokens(tokens, n)
        h[n:2 * n] = p
        h[2 * n:3 * n] = table[p // bs] * bs + p % bs
        h[3 * n:] = table
        d = host.to(self.e.device, non_blocking=True)
        return d[:n], d[n:2 * n], d[2 * n:3 * n], d[3 * n:]

    @staticmethod
    def _places(rows: Sequence[int], n: int) -> List[int]:
        """The rows as places among n.  (Checked here: a slice ends where there are no more rows, and the kernels that pick rows read where they are told.)"""
        rows = [index(r) for r in rows]
        for r in rows:
            if not -n <= r < n:
                raise IndexError("row %d is not among %d tokens" % (r, n))
        return [r + n if r < 0 else r for r in rows]

    @staticmethod
    def _run_of(rows: Sequence[int]) -> Optional[slice]:
        """The rows as a slice, if they are one after another."""
        r = list(rows)
        return slice(r[0], r[-1] + 1) if r and r[0] >= 0 and r == list(range(r[0], r[-1] + 1)) else None

    @staticmethod
    def _splits_for(ctas: int, keys: int) -> int:
        """Splits of the key range per (sequence, KV head): about four CTAs per SM, at least 256 keys per split."""
        return max(1, min(32, keys // 256, (148 * 4 + ctas - 1) // max(ctas, 1)))


class Sampler:
    """Temperature / top-k / nucleus sampling of next tokens from logits [rows, vocab] with its own random generator, so
    that a run is reproducible from its seed.  `temperature == 0` (or `top_k == 1`) is greedy."""

    def __init__(self, temperature: float = 1.0, top_k: int = 0, top_p: float = 1.0, seed: int = 0, device="cpu"):
        self.temperature, self.top_k, self.top_p = float(temperature), int(top_k), float(top_p)
        self.gen = torch.Generator(device=device).manual_seed(int(seed))

    def __call__(self, logits: torch.Tensor) -> torch.Tensor:
        if self.temperature <= 0.0 or self.top_k == 1:
            return logits.argmax(-1)
        z = logits / self.temperature
        if self.top_k > 0 and self.top_k < z.shape[-1]:
            kth = z.topk(self.top_k, -1).values[..., -1:]
            z = z.masked_fill(z < kth, float("-inf"))
        if self.top_p < 1.0:
            order = z.sort(-1, descending=True)
            p = torch.softmax(order.values, -1)
            before = p.cumsum(-1) - p                     # probability mass ahead of each token, in sorted order
            drop = before >= self.top_p                   # the first token always stays
            z = z.masked_fill(torch.zeros_like(drop).scatter(-1, order.indices, drop), float("-inf"))
        return torch.multinomial(torch.softmax(z, -1), 1, generator=self.gen).squeeze(-1)


@torch.no_grad()
def generate(engine, prompts: Sequence[Sequence[int]], max_new_tokens: int, *, temperature: float = 0.0,
             top_k: int = 0, top_p: float = 1.0, seed: int = 0, eos_id: int = -1, block_size: int = 16,
             max_num_seqs: int = 64, max_num_batched_tokens: int = 4096, kv_dtype=None,
             prefix_cache_bytes: int = 0) -> List[List[int]]:
    """Continue every prompt by up to `max_new_tokens` tokens (stopping at `eos_id`) with continuous batching on a paged KV
    cache sized for the request, and return the new tokens per prompt.  Greedy by default (the decode step is replayed
    from CUDA graphs on a GPU); with `temperature > 0` the next tokens are drawn by `Sampler` (eager decode steps).
    `engine`: any engine of `models.registry`."""
    from ..serving import Request, ServingScheduler
    from .registry import new_serving
    need = sum((len(p) + max_new_tokens + block_size - 1) // block_size for p in prompts)
    greedy = temperature <= 0.0 or top_k == 1
    model = new_serving(engine, num_blocks=need + 1, block_size=block_size, max_num_seqs=max_num_seqs, kv_dtype=kv_dtype,
                        graphs=greedy, prefix_cache_bytes=prefix_cache_bytes)  # prompts of one call that share a prefix reuse its blocks
    if not greedy:
        model.sampler = Sampler(temperature, top_k, top_p, seed, device=engine.device)
    sched = ServingScheduler(num_blocks=need + 1, block_size=block_size, max_num_seqs=max_num_seqs,
                             max_num_batched_tokens=max_num_batched_tokens, eos_id=eos_id)
    limit = engine.cfg.max_seq                            # None: the model's positions have no end
    reqs = [Request(i, list(p), max_new_tokens=max_new_tokens) for i, p in enumerate(prompts)]
    for r in reqs:
        if limit and len(r.prompt_tokens) + max_new_tokens > limit:
            raise ValueError("prompt %d: %d tokens + %d new exceed the model's %d positions" %
                             (r.id, len(r.prompt_tokens), max_new_tokens, limit))
        sched.add_request(r)
    finished, guard = 0, 0
    while finished < len(reqs):
        finished += len(sched.step(model))
        guard += 1
        if guard > 4 * (max_new_tokens + len(reqs)) + 64 + sum(len(p) for p in prompts):
            raise RuntimeError("the schedule did not finish")
    return [list(r.generated_tokens) for r in reqs]
