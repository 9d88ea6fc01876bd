"""Chunked prompt processing for a MiniCPM3 decode session (latent cache).

The reference walks a prompt one token at a time (``tests/models/orchestrator/causal_lm/generation.py:56-61``).
Here consecutive prompt tokens go through the layer stack together, up to 4096 of them: every projection streams its
weights once per chunk on the tensor cores; for the chunk's attention every head's keys and values are expanded from the
latents of the context (to f32 accuracy, as two bf16 terms), so that it runs as causal flash attention.  The cache rows
and the position the session ends with are those of the token-by-token walk.
"""
from __future__ import annotations

import ctypes as C
import weakref

import torch

from .. import lib
from . import paged_kv

CHUNK = 4096


class MiniCPM3Prefill:
    def __init__(self, sess):
        cfg, dev = sess.cfg, sess.device
        self.sess = weakref.proxy(sess)                  # (no cycle: a session and its graph go when their owner lets go)
        H, I, NH, VD = cfg.hidden_size, cfg.intermediate_size, cfg.num_attention_heads, cfg.v_head_dim
        NOPE, R, KVL, QL = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.kv_lora_rank, cfg.q_lora_rank
        #: tokens of one chunk: no more scratch than the session's capacity can use
        self.chunk = M = max(2, min(CHUNK, sess.max_ctx))
        scratch = lambda *s: torch.empty(*s, device=dev, dtype=torch.bfloat16)
        self.hidden, self.norm = scratch(M, H), scratch(M, H)
        self.qkv_a, self.attn, self.act = scratch(M, QL + KVL + R), scratch(M, NH * VD), scratch(M, I)
        self.qa, self.q = scratch(M, QL), scratch(M, NH * (NOPE + R))
        self.lat = scratch(sess.max_ctx, KVL)
        self.kv_hi, self.kv_lo = (scratch(sess.max_ctx, NH * (NOPE + VD)) for _ in range(2))
        self.status = torch.zeros(1, device=dev, dtype=torch.int32)
        self.positions = torch.arange(sess.max_ctx, device=dev, dtype=torch.int32)
        a = sess.args
        self.args = lib.MiniCPM3PrefillArgs(
            layers=sess._layer_structs, n_layers=len(sess.layers), m=M, hidden=H, heads=NH, q_lora=QL, kv_lora=KVL,
            nope=NOPE, rope=R, v=VD, inter=I, vocab=cfg.vocab_size, eps=a.eps, lora_eps=a.lora_eps, scale=a.scale,
            embed_scale=a.embed_scale, residual_scale=a.residual_scale, pdl=a.pdl, w_embed=lib.ptr(sess.w_embed),
            cos_table=lib.ptr(sess.cos), sin_table=lib.ptr(sess.sin), max_pos=sess.max_pos, page_size=paged_kv.PAGE_SIZE,
            table_len=sess.table.shape[1], max_ctx=sess.max_ctx, block_table=lib.ptr(sess.table), ids=None, pos_rows=None,
            hidden_buf=lib.ptr(self.hidden), norm_buf=lib.ptr(self.norm), qkv_a_buf=lib.ptr(self.qkv_a),
            attn_buf=lib.ptr(self.attn), act_buf=lib.ptr(self.act), status=lib.ptr(self.status), qa_buf=lib.ptr(self.qa),
            lat_buf=lib.ptr(self.lat), q_buf=lib.ptr(self.q), kv_hi_buf=lib.ptr(self.kv_hi), kv_lo_buf=lib.ptr(self.kv_lo))

    def launches(self, m: int) -> int:
        """Kernels one chunk enqueues: embed + per layer 2 norms, 6 projections, 3 of the attention."""
        return 1 + 11 * len(self.sess.layers)

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
            self.args.m, self.args.first = m, start
            self.args.pos_rows = self.positions.data_ptr() + 4 * start
            self.args.ids = sess.tokens.data_ptr() + 8 * start
            lib.check(lib.load().tfb_minicpm3_prefill_chunk(C.byref(self.args), lib.stream()), "tfb_minicpm3_prefill_chunk")
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
