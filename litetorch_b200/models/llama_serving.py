"""KV-cache serving on the Llama engine's weights: chunked prefill into a paged cache, batched one-token decode on
the split-K paged attention kernel, greedy sampling on the device.

`LlamaKVModel` is the model side of `serving.ServingScheduler.step`: the native scheduler (admission, block tables,
chunked prefill within a token budget, completion) hands it prompt chunks and the running sequences' newest tokens
together with their block tables, and gets next tokens back.  Nothing is recomputed: every token's K and V are
written once (`lt_rope_append`, with the rotation of queries and keys) and read by the attention of later tokens (`lt_paged_decode`, `lt_flash_fwd` for a
prompt chunk).  The reference's counterparts: ContinuousBatchingScheduler::step and its block tables
(src/llm/continuous_batching.cpp:20-197), paged attention (src/ops/attention.cpp:351-477) and flash-decoding
(src/ops/flash_decoding.cpp:13-115); its cache is never filled.
"""
from __future__ import annotations

from collections import OrderedDict
from typing import List, Sequence

import numpy as np
import torch

from ..serving import PagedKVCache
from .llama import LlamaEngine
from .serving_base import Sampler, ServingModel, _ints, generate          # noqa: F401  (their names live here as well)


class LlamaKVModel(ServingModel):
    def __init__(self, engine: LlamaEngine, num_blocks: int, block_size: int = 16, kv_dtype=torch.bfloat16, num_splits: int = 0,
                 graphs: bool = True, prefix_cache_bytes: int = 0):
        assert engine.w.tp == 1 and hasattr(engine.w, "flat_p"), "serving runs on whole (unsharded) weights"
        super().__init__(engine, block_size, graphs)
        cfg = engine.cfg
        self.num_splits = num_splits
        self.cache = PagedKVCache(cfg.n_layers, num_blocks, block_size, cfg.n_kv_heads, cfg.head_dim, device=engine.device,
                                  dtype=kv_dtype)
        self.kv_bytes_per_token = 2 * cfg.n_layers * cfg.n_kv_heads * cfg.head_dim * self.cache.k[0].element_size()
        # ---- prefix reuse: K / V of finished prompts' whole blocks are kept as snapshots (up to `prefix_cache_bytes`,
        # least recently used first out); a later prompt that starts with the same tokens gets those blocks by a copy
        # and only its remaining tokens are computed.  The reference has the prefix map (src/llm/prefix_cache.cpp) but
        # never consults it while serving.
        self.prefix_cache_bytes = int(prefix_cache_bytes)
        self._snap = OrderedDict()           # handle -> (k [layers, nb, Hkv, bs, hd], v, bytes)
        self._snap_bytes = 0
        self._next_handle = 1
        self._seq_tokens = {}                # first block of a sequence in prefill -> its prompt tokens so far
        if self.prefix_cache_bytes > 0:
            from ..serving import PrefixCache
            self._index = PrefixCache()

    def _tokens(self, tokens, n):
        # the embedding takes a token past the vocabulary for the nearest one it has, one past 32 bits too
        try:
            return super()._tokens(tokens, n)
        except OverflowError:
            return np.clip(_ints(tokens, n, np.int64), -1 << 31, (1 << 31) - 1)

    # ------------------------------------------------------------------ shared layer body
    def _layers(self, x, attend):
        """attend(i, qkv) of a layer's unrotated rows [q | k | v] writes their keys and values to the cache; its result joins x."""
        e, cfg, w, K = self.e, self.e.cfg, self.e.w, self.e.K
        n = x.shape[0]
        for i in range(cfg.n_layers):
            p = "layers.%d." % i
            qkv = K.product_of_constants(x, w.p(p + "wqkv"), norm=(w.p(p + "attn_norm"), cfg.rms_eps))
            o = attend(i, qkv)
            x1 = K.product_of_constants(o.reshape(n, -1), w.p(p + "wo"), residual=x)
            hm = K.product_of_constants(x1, w.p(p + "w_gu"), act="silu", norm=(w.p(p + "mlp_norm"), cfg.rms_eps))
            x = K.product_of_constants(hm, w.p(p + "w_down"), residual=x1)
        return x

    def _logits(self, hidden, rows=None):
        e, K = self.e, self.e.K
        if rows is not None:
            run = self._run_of(rows)
            hidden = hidden[rows if run is None else run]
        return K.product_of_constants(hidden, e.w.p("lm_head"), norm=(e.w.p("final_norm"), e.cfg.rms_eps))

    # ------------------------------------------------------------------ prompt chunks
    @torch.no_grad()
    def prefill_chunk(self, tokens: Sequence[int], start: int, block_ids: Sequence[int], want_token: bool, slot: int = 0) -> int:
        """Run prompt positions [start, start + len(tokens)) of one sequence: their K / V go into the sequence's blocks,
        their queries attend to everything cached so far.  Returns the next token when `want_token` (the chunk completes
        the prompt), else -1."""
        if self.prefix_cache_bytes > 0:
            return self._prefill_with_reuse(list(tokens), start, block_ids, want_token)
        return super().prefill_chunk(tokens, start, block_ids, want_token)

    # ---- prefix reuse around the computation
    def _prefill_with_reuse(self, tokens: List[int], start: int, block_ids: Sequence[int], want_token: bool) -> int:
        bs = self.block_size
        key = block_ids[0]
        sofar = (self._seq_tokens.get(key, []) if start > 0 else []) + tokens
        end = start + len(tokens)
        matched, handles = self._index.longest_prefix(sofar, bs)
        snap = self._snap.get(handles[0]) if handles else None
        covered = start
        if snap is not None and matched > start:
            self._snap.move_to_end(handles[0])
            m = min(matched, snap[0].shape[1] * bs)
            if m >= end and want_token:                           # the last token's logits are needed: compute it
                m = (end - 1) // bs * bs
            if m > start:
                b0, b1 = start // bs, m // bs
                dst = torch.tensor(list(block_ids[b0:b1]), dtype=torch.int64, device=self.e.device)
                for i in range(self.e.cfg.n_layers):
                    self.cache.k[i][dst] = snap[0][i, b0:b1]
                    self.cache.v[i][dst] = snap[1][i, b0:b1]
                self.prefill_tokens_reused += m - start
                covered = m
        out = super().prefill_chunk(sofar[covered:end], covered, block_ids, want_token) if covered < end else -1
        if want_token:
            self._seq_tokens.pop(key, None)
            self._remember(sofar, block_ids)
        else:
            self._seq_tokens[key] = sofar
        return out

    def _remember(self, prompt: List[int], block_ids: Sequence[int]) -> None:
        bs = self.block_size
        nb = len(prompt) // bs
        if nb == 0:
            return
        L = nb * bs
        got, handles = self._index.longest_prefix(prompt[:L], bs)
        if got == L and handles and handles[0] in self._snap:
            return                                                # this prefix is cached already
        blocks = torch.tensor(list(block_ids[:nb]), dtype=torch.int64, device=self.e.device)
        k = torch.stack([self.cache.k[i][blocks] for i in range(self.e.cfg.n_layers)])
        v = torch.stack([self.cache.v[i][blocks] for i in range(self.e.cfg.n_layers)])
        nbytes = 2 * k.numel() * k.element_size()
        if nbytes > self.prefix_cache_bytes:
            return
        while self._snap and self._snap_bytes + nbytes > self.prefix_cache_bytes:
            _, (_, _, old) = self._snap.popitem(last=False)
            self._snap_bytes -= old
        h = self._next_handle
        self._next_handle += 1
        self._snap[h] = (k, v, nbytes)
        self._snap_bytes += nbytes
        # findable by prompts that share the whole thing or a power-of-two number of its blocks: a later prompt reuses at
        # least half of the whole blocks it shares, for a logarithmic number of index entries per prompt
        lengths, j = {L}, 1
        while j * bs < L:
            lengths.add(j * bs)
            j *= 2
        from ..serving import _i32
        for n in sorted(lengths):                                 # the native index alone (it evicts by itself)
            self._index._lib.lt_prefix_insert(self._index._c, _i32(prompt[:n]), n, _i32([h]), 1)

    def _prompt_hidden(self, tokens: Sequence[int], start: int, block_ids: Sequence[int], slot: int = 0):
        e, K = self.e, self.e.K
        dev = e.device
        n = len(tokens)
        tok, pos, slots, blocks = self._prompt_inputs(tokens, start, block_ids)
        bs = self.block_size
        Hq, Hkv, hd = e.cfg.n_heads, e.cfg.n_kv_heads, e.cfg.head_dim

        def attend(i, qkv):
            # a first portion attends to its own rows, rotated in place; a later one to the cache, for which its queries are packed
            q = K.rope_append(qkv, e.cos, e.sin, pos, slots, Hq, Hkv, hd, self.cache.k[i], self.cache.v[i], bs, self.cache.fp8, self.cache.k_scale,
                              self.cache.v_scale, in_place=start == 0)
            k = qkv[:, Hq * hd:(Hq + Hkv) * hd].view(n, Hkv, hd)
            v = qkv[:, (Hq + Hkv) * hd:(Hq + 2 * Hkv) * hd].view(n, Hkv, hd)
            if start == 0:
                o, _ = K.flash_fwd(q.unsqueeze(0), k.unsqueeze(0), v.unsqueeze(0), causal=True)
                return o[0]
            # later chunk: keys and values of the whole context so far, read back from the sequence's blocks
            kc, vc = torch.empty(2, start + n, Hkv, hd, dtype=self.cache.k[i].dtype, device=dev)
            K.kv_gather(self.cache.k[i], self.cache.v[i], blocks, 0, start + n, kc, vc)
            if self.cache.fp8:
                kc = (kc.float() * self.cache.k_scale).to(q.dtype)
                vc = (vc.float() * self.cache.v_scale).to(q.dtype)
            o, _ = K.flash_fwd(q.unsqueeze(0), kc.unsqueeze(0), vc.unsqueeze(0), causal=True)
            return o[0]

        return self._layers(K.embedding_fwd(tok, e.w.p("embed")), attend)

    # ------------------------------------------------------------------ one token for every running sequence
    def _decode_hidden(self, d: torch.Tensor, S: int, width: int) -> torch.Tensor:
        e, K = self.e, self.e.K
        cfg, c, bs = e.cfg, self.cache, self.block_size
        tok, pos, slots, ctx = d[0], d[1], d[2], d[3]
        bt = d[5:].t().contiguous()

        def attend(i, qkv):
            # early: the tables were made, and what earlier passes cached was complete, before the embedding, which starts after everything before it
            return K.decode_step(qkv, e.cos, e.sin, pos, slots, cfg.n_heads, cfg.n_kv_heads, cfg.head_dim, c.k[i], c.v[i], bt, ctx, bs, self.num_splits, c.k_scale, c.v_scale,
                                 early=True)

        return self._layers(K.embedding_fwd(tok, e.w.p("embed")), attend)
