"""Chunked prompt processing for a Qwen3.5 decode session.

The reference walks a prompt one token at a time (``tests/models/orchestrator/causal_lm/generation.py:56-61``).
Here up to 512 consecutive prompt tokens go through the layer stack together: projections and touched experts are read
once per chunk, the Gated DeltaNet state walks the tokens in order inside one kernel.  State, windows, cache rows and
the position the session ends with are those of the token-by-token walk.
"""
from __future__ import annotations

import ctypes as C
import weakref

import torch

from .. import lib

CHUNK = 512


class Qwen35Prefill:
    def __init__(self, sess):
        cfg, dev = sess.cfg, sess.device
        self.sess = weakref.proxy(sess)                  # (no cycle: a session and its graph go when their owner lets go)
        self.chunk = M = max(2, min(CHUNK, sess.max_ctx))
        H, E, K, I = cfg.hidden, cfg.n_experts, cfg.top_k, cfg.moe_intermediate
        QD, KD, VD = cfg.n_q_heads * cfg.head_dim, cfg.key_dim, cfg.val_dim
        widest = max(cfg.conv_dim + VD + 2 * cfg.gdn_n_v_heads, 2 * QD + 2 * cfg.n_kv_heads * cfg.head_dim)
        f32, bf, i32, i64 = torch.float32, torch.bfloat16, torch.int32, torch.int64
        shapes = dict(hidden=(f32, M, H), attended=(f32, M, H), normed=(f32, M, H), norm16=(bf, M, H), proj=(bf, M, widest),
                      mixed=(bf, M, max(VD, QD)), out16=(bf, M, H), qk=(f32, M, max(2 * KD, QD)), v=(f32, M, VD),
                      read=(f32, M, VD), gates=(f32, M, cfg.gdn_n_v_heads, 2), logits=(f32, M, E + 1), indices=(i64, M, K),
                      weights=(f32, M, K), shared_gate=(f32, M), inner=(bf, M, K + 1, I), y=(bf, M, K + 1, H),
                      counts=(i32, 2 * (E + 1) + 1), lists=(i32, E + 1, M))
        self.scratch = {n: torch.empty(*s, device=dev, dtype=dt) for n, (dt, *s) in shapes.items()}
        self.status = torch.zeros(1, device=dev, dtype=i32)
        self.positions = torch.arange(sess.max_ctx, device=dev, dtype=i32)
        self.args = lib.Qwen35PrefillArgs(step=C.pointer(sess.args), status=lib.ptr(self.status), pdl=sess.args.pdl,
                                          **{n: lib.ptr(t) for n, t in self.scratch.items()})

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
            lib.check(lib.load().tfb_qwen35_prefill_chunk(C.byref(self.args), lib.stream()), "tfb_qwen35_prefill_chunk")
            done += m
        if pick and done == n_tokens:
            sess.pos.fill_(first + done - 1)
            return self.scratch["hidden"][m - 1].data_ptr()
        sess.pos.fill_(first + done)
        for _ in range(n_tokens - done):                 # a lone leftover token takes the ordinary step
            sess.step()

    def check_status(self) -> None:
        code = int(self.status.item())
        if code:
            self.status.zero_()                          # told once
            raise RuntimeError(f"a bounded wait of a prompt chunk's kernels gave up (status {code:#x})")
