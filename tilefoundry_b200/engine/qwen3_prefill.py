"""Chunked prompt processing for a Qwen3 decode session.

The reference walks a prompt one token at a time (``tests/models/orchestrator/causal_lm/generation.py:56-61``).
Here consecutive prompt tokens go through the layer stack together, up to 4096 of them: every projection streams its
weights once per chunk on the tensor cores, and attention runs in its chunk form (each token attends to the cached rows
before it).  The cache rows and the position the session ends with are those of the token-by-token walk.
"""
from __future__ import annotations

import ctypes as C
import weakref
import torch

from .. import lib
from . import paged_kv


class Qwen3Prefill:
    def __init__(self, sess):
        cfg, dev = sess.cfg, sess.device
        self.sess = weakref.proxy(sess)                  # (no cycle: a session and its graph go when their owner lets go)
        HQ, HKV, D, H, I = (cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.hidden_size,
                            cfg.intermediate_size)
        bf, f32, i32 = torch.bfloat16, torch.float32, torch.int32
        most = lib.load().tfb_qwen3_prefill_max_chunk(H, HQ, HKV, D, I, paged_kv.PAGE_SIZE)
        #: tokens of one chunk: what the kernels take, and no more scratch than the session's capacity can use
        self.chunk = M = max(2, min(most, sess.max_ctx))
        scratch = lambda *s, dtype=bf: torch.empty(*s, device=dev, dtype=dtype)
        self.hidden, self.norm = scratch(M, H), scratch(M, H)
        self.qkv, self.attn, self.act = scratch(M, (HQ + 2 * HKV) * D), scratch(M, HQ * D), scratch(M, I)
        self.part_o = self.part_ml = self.counters = None
        if most <= 32:                                   # attention split per token: scratch for the partials
            nsplit = lib.attn_splits(sess.max_ctx)
            self.part_o = scratch(M * HQ * nsplit * D, dtype=f32)
            self.part_ml = scratch(M * HQ * nsplit * 2, dtype=f32)
            self.counters = torch.zeros(M * HKV, device=dev, dtype=i32)
        self.status = torch.zeros(1, device=dev, dtype=i32)
        self.positions = torch.arange(sess.max_ctx, device=dev, dtype=i32)
        self._layers = (lib.Qwen3BatchLayer * len(sess.layers))()
        for s, layer in zip(self._layers, sess.layers):
            for name, _ in lib.Qwen3BatchLayer._fields_:
                setattr(s, name, lib.ptr(layer[name]))
        a = sess.args
        self.args = lib.Qwen3PrefillArgs(
            layers=self._layers, n_layers=len(sess.layers), m=M, hidden=H, hq=HQ, hkv=HKV, d=D, inter=I,
            pdl=a.pdl, eps=a.eps, scale=a.scale, vocab=cfg.vocab_size, w_embed=lib.ptr(sess.w_embed),
            cos_table=lib.ptr(sess.cos), sin_table=lib.ptr(sess.sin), max_pos=sess.max_pos,
            page_size=paged_kv.PAGE_SIZE, table_len=sess.table.shape[1], max_ctx=sess.max_ctx,
            block_table=lib.ptr(sess.table), ids=None, pos_rows=None,
            hidden_buf=lib.ptr(self.hidden), norm_buf=lib.ptr(self.norm), qkv_buf=lib.ptr(self.qkv),
            attn_buf=lib.ptr(self.attn), act_buf=lib.ptr(self.act), part_o=lib.ptr(self.part_o),
            part_ml=lib.ptr(self.part_ml), counters=lib.ptr(self.counters), status=lib.ptr(self.status))
        #: kernels one chunk enqueues (embed + 8 per layer)
        self.launches_per_chunk = 1 + 8 * len(sess.layers)

    def run(self, n_tokens: int, first: int | None = None, pick: bool = False) -> int | None:
        """Positions ``pos .. pos + n_tokens - 1`` of the session's token history; *first*: the position, where the
        caller knows it (else it is read from the device).  *pick*: the caller picks the token after the last of them: the
        position stays at that last one and the address of its hidden state is returned (None where a step took it)."""
        sess = self.sess
        first = int(sess.pos.item()) if first is None else first
        if n_tokens < 0 or first + n_tokens > sess.max_ctx:
            raise ValueError(f"{first}+{n_tokens} tokens exceed capacity {sess.max_ctx}")
        sess.prompt_unchecked = True
        done = 0
        while n_tokens - done >= 2:
            m = min(self.chunk, n_tokens - done)
            if n_tokens - done - m == 1 and m > 2:       # never leave a single token: a chunk holds at least two
                m -= 1
            start = first + done
            self.args.m = m
            self.args.ids = sess.tokens.data_ptr() + 8 * start
            self.args.pos_rows = self.positions.data_ptr() + 4 * start
            lib.check(lib.load().tfb_qwen3_prefill_chunk(C.byref(self.args), lib.stream()), "tfb_qwen3_prefill_chunk")
            done += m
        if pick and done == n_tokens:
            sess.pos.fill_(first + done - 1)
            return self.hidden[m - 1].data_ptr()
        sess.pos.fill_(first + done)
        for _ in range(n_tokens - done):                 # a lone leftover token takes the ordinary step
            sess.step()

    def check_status(self) -> None:
        code = int(self.status.item())
        if code:
            self.status.zero_()                          # told once
            raise RuntimeError(f"a bounded wait of a prompt chunk's kernels gave up (status {code})")
