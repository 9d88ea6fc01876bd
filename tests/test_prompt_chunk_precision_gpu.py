"""Error of a prompt chunk's kernels against 64 bits, beside that of the one-token (or 32-token) kernels on the same inputs:
where tensor cores and two-term bf16 operands stand in for f32 multiply-adds, the results are no further off."""
import ctypes as C
from dataclasses import replace

import pytest
import torch

from tilefoundry_b200.authored import minicpm3_4b as mc
from tilefoundry_b200.authored import qwen3_1_7b as q
from tilefoundry_b200.authored.weights import random_weights_on
from tilefoundry_b200.runtime import DictResource

pytestmark = pytest.mark.gpu
BF, DEV = torch.bfloat16, "cuda:0"
# Both sides round their outputs to bf16, 1.6e-3 of the norm.  An error of 2^-16 before that rounding adds (2^-16 / 1.6e-3)^2 / 2 =
# 5e-5 to it, and the few hundredths of a per cent of elements that fall on the other side of a midpoint move it by 1e-4: a
# form that is further off by more than this share has lost bits.
SHARE = 1.0005


@pytest.fixture(scope="module")
def so():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tilefoundry_b200 import lib
    return lib.load()


def _error(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


def _no_worse(name, new, old, want):
    """*new* and *old* bf16 outputs, *want* in 64 bits; also counts the elements that are not the nearest bf16."""
    e_new, e_old = _error(new, want), _error(old, want)
    off = [(x != want.to(torch.float32).to(BF)).double().mean().item() for x in (new, old)]
    print(f"{name}: error {e_new:.6e} (before {e_old:.6e}), not the nearest bf16 {off[0]:.2e} (before {off[1]:.2e})")
    assert e_new <= e_old * SHARE, name


def _rotate(x, cos, sin):
    """x [m, heads, d] bf16 -> rotated, one rounding (f64 products, exact for bf16 factors, and their f32 sum)."""
    d = x.shape[-1]
    other = torch.cat([-x[..., d // 2:], x[..., : d // 2]], -1)
    return (x.float() * cos.float()[:, None] + other.float() * sin.float()[:, None]).to(BF)


def _attend(qs, k, v, first):
    """Causal attention in 64 bits: qs [m, heads, dk] already scaled, k and v [positions, heads, .]."""
    out = torch.empty(qs.shape[0], qs.shape[1], v.shape[-1], dtype=torch.float64, device=DEV)
    mask = torch.arange(k.shape[0], device=DEV)[None] > first + torch.arange(qs.shape[0], device=DEV)[:, None]
    for h in range(qs.shape[1]):
        s = (qs[:, h].double() @ k[:, h].double().t()).masked_fill(mask, -float("inf"))
        out[:, h] = torch.softmax(s, -1) @ v[:, h].double()
    return out


@pytest.mark.parametrize("n,first,gain", [(64, 0, 1.0), (300, 0, 1.0), (257, 700, 1.0), (1500, 0, 3.0), (4093, 0, 1.0)])
def test_grouped_query_attention(so, n, first, gain):
    from tilefoundry_b200 import lib
    from tilefoundry_b200.engine.qwen3 import Qwen3Session
    cfg = replace(q.QWEN3_1_7B, num_hidden_layers=1, vocab_size=2048)
    HQ, HKV, D = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    w = random_weights_on(q.build(cfg), DEV, seed=3, std=0.02)
    sess = Qwen3Session(cfg, DictResource(w), max_ctx=-(-(first + n) // 64) * 64, device=DEV)
    L, g = sess.layers[0], torch.Generator(device=DEV).manual_seed(n)
    for t in (L["gamma_q"], L["gamma_k"]):
        t.copy_(gain * (1 + 0.1 * torch.randn(D, device=DEV, generator=g)))
    sess.reset(torch.randint(0, cfg.vocab_size, (first + n,), generator=torch.Generator().manual_seed(n)))
    rows = lambda pool: pool.view(-1, HKV, D)
    rows(L["k_pool"])[:first].normal_(generator=g)
    rows(L["v_pool"])[:first].normal_(generator=g)
    sess.pos.fill_(first)
    sess.prefill(n)
    sess.check_prompt()
    pre = sess._prefill
    new = pre.attn[:n].view(n, HQ, D).clone()
    k, v = rows(L["k_pool"])[: first + n].clone(), rows(L["v_pool"])[: first + n].clone()
    qs = pre.qkv[:n].view(n, HQ + 2 * HKV, D)[:, :HQ].clone()       # normalised, rotated, scaled: bf16 in either form
    # the same q | k | v rows again, and the form that the decode steps' kernel takes them in
    x = sess.w_embed[sess.tokens[first: first + n]].contiguous()
    lib.check(so.tfb_rmsnorm(lib.ptr(x), lib.ptr(L["gamma_in"]), lib.ptr(pre.norm), n, cfg.hidden_size, sess.args.eps,
                             lib.NORM_CAST_THEN_GAIN, lib.stream()), "tfb_rmsnorm")
    gemm = lib.GemmSmallMArgs(w=lib.ptr(L["w_qkv"]), x=lib.ptr(pre.norm), y=lib.ptr(pre.qkv), status=lib.ptr(pre.status), m=n,
                              n=(HQ + 2 * HKV) * D, k=cfg.hidden_size)
    lib.check(so.tfb_gemm_rows(C.byref(gemm), lib.stream()), "tfb_gemm_rows")
    assert torch.equal(pre.qkv[:n].view(n, -1, D)[:, HQ + HKV:], v[first:])
    nsplit = lib.attn_splits(sess.max_ctx)
    old = torch.empty(n, HQ, D, device=DEV, dtype=BF)
    f32 = lambda *s: torch.zeros(*s, device=DEV)
    for lo in range(0, n, 512):                                     # (a few hundred MB of split results at a time)
        m = min(512, n - lo)
        part_o, part_ml, counters = f32(m * HQ * nsplit * D), f32(m * HQ * nsplit * 2), torch.zeros(m * HKV, device=DEV, dtype=torch.int32)
        pos = torch.arange(first + lo, first + lo + m, device=DEV, dtype=torch.int32)
        for chunk in (1, 2):
            a = lib.AttnGqaArgs(qkv=lib.ptr(pre.qkv[lo]), gamma_q=lib.ptr(L["gamma_q"]), gamma_k=lib.ptr(L["gamma_k"]), cos_table=lib.ptr(sess.cos),
                                sin_table=lib.ptr(sess.sin), pos=lib.ptr(pos), k_pool=lib.ptr(L["k_pool"]), v_pool=lib.ptr(L["v_pool"]),
                                block_table=lib.ptr(sess.table), out=lib.ptr(old[lo]), part_o=lib.ptr(part_o), part_ml=lib.ptr(part_ml),
                                counters=lib.ptr(counters), hq=HQ, hkv=HKV, d=D, rotary_dim=D, page_size=64, table_len=sess.table.shape[1],
                                max_ctx=sess.max_ctx, max_pos=sess.max_pos, eps=sess.args.eps, scale=sess.args.scale,
                                norm_mode=lib.NORM_CAST_THEN_GAIN, pdl=0, batch=m, chunk=chunk)
            lib.check(so.tfb_attn_gqa_decode(C.byref(a), lib.stream()), "tfb_attn_gqa_decode")
    torch.cuda.synchronize()
    _no_worse(f"attention, {n} tokens from {first}, gain {gain}", new, old,
              _attend(qs, k.repeat_interleave(HQ // HKV, 1), v.repeat_interleave(HQ // HKV, 1), first))


@pytest.mark.parametrize("n,std", [(64, 0.02), (512, 0.02), (1024, 0.05)])
def test_latent_attention(so, n, std):
    from tilefoundry_b200 import lib
    from tilefoundry_b200.engine.minicpm3 import MiniCPM3Session
    cfg = replace(mc.MINICPM3_4B, num_hidden_layers=1, vocab_size=2048)
    NH, QL, KVL, NOPE, R, VD = (cfg.num_attention_heads, cfg.q_lora_rank, cfg.kv_lora_rank, cfg.qk_nope_head_dim, cfg.qk_rope_head_dim,
                                cfg.v_head_dim)
    w = random_weights_on(mc.build(cfg), DEV, seed=4, std=std)
    sess = MiniCPM3Session(cfg, DictResource(w), max_ctx=n, device=DEV)
    L, a = sess.layers[0], sess.args
    sess.reset(torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(n)))
    sess.prefill(n)
    sess.check_prompt()
    pre = sess._prefill

    def reference(qkv_a, qs=None):
        """The authored rounding points up to the scaled query (or the query that the form itself rounded: which side of a
        midpoint a sum falls on is the projection's error, below), then 64 bits from the cached latents."""
        c = qkv_a[:, :QL].double()
        c = (c * torch.rsqrt(c.square().mean(-1, keepdim=True) + cfg.lora_eps)).to(torch.float32).to(BF)
        qa = (c.float() * L["gamma_q_a"].float()).to(BF)
        qh = (qa.double() @ L["w_q_b"].double().t()).to(torch.float32).to(BF).view(n, NH, NOPE + R)
        scaled = lambda t: (t.float() * a.scale).to(BF)
        rope = _rotate(qh[..., NOPE:], sess.cos[:n], sess.sin[:n])
        mine = torch.cat([scaled(qh[..., :NOPE]), scaled(rope)], -1)
        if qs is not None:
            assert (qs != mine).double().mean() < 2e-3 and (qs.float() - mine.float()).abs().max() <= 2 ** -7 * mine.float().abs().max()
            mine = qs
        cached = L["k_pool"].view(-1, KVL + R)[:n]
        kv = (cached[:, :KVL].double() @ L["w_kv_b"].double().t()).view(n, NH, NOPE + VD)
        k = torch.cat([kv[..., :NOPE], cached[:, None, KVL:].double().expand(n, NH, R)], -1)
        return _attend(mine, k, kv[..., NOPE:], 0)
    new, want_new = pre.attn[:n].view(n, NH, VD).clone(), reference(pre.qkv_a[:n], pre.q[:n].view(n, NH, NOPE + R))
    # the form of up to 32 tokens: queries absorbed to f32, attention over the latents in f32
    nsplit = so.tfb_mla_latent_splits(sess.max_ctx)
    f32 = lambda *s: torch.zeros(*s, device=DEV)
    scratch = dict(q_lat_buf=f32(32, NH * 2 * KVL), q_rope_buf=f32(32, NH * R), part_o=f32(32, NH * nsplit * KVL), part_ml=f32(32, NH * nsplit * 2))
    args = type(pre.args).from_buffer_copy(pre.args)
    args.qa_buf, args.m = None, 32
    for name, t in scratch.items():
        setattr(args, name, lib.ptr(t))
    old, qkv_a = torch.empty_like(new), torch.empty_like(pre.qkv_a[:n])
    for lo in range(0, n, 32):
        args.ids, args.pos_rows = sess.tokens.data_ptr() + 8 * lo, pre.positions.data_ptr() + 4 * lo
        lib.check(so.tfb_minicpm3_prefill_chunk(C.byref(args), lib.stream()), "tfb_minicpm3_prefill_chunk")
        old[lo: lo + 32], qkv_a[lo: lo + 32] = pre.attn[:32].view(32, NH, VD), pre.qkv_a[:32]
    sess.check_prompt()
    want_old = reference(qkv_a)
    e_new, e_old = _error(new, want_new), _error(old, want_old)
    print(f"latent attention, {n} tokens, std {std}: error {e_new:.6e} (before {e_old:.6e})")
    assert e_new <= e_old * SHARE


# the input and output projections of the f32-activation family, Qwen3's, and the low-rank query's
@pytest.mark.parametrize("m,n,k", [(512, 3840, 768), (64, 12352, 2048), (300, 9216, 2048), (512, 2048, 4096), (33, 4096, 2048), (1500, 2048, 6144)])
def test_projections(so, m, n, k):
    from tilefoundry_b200 import lib
    g = torch.Generator(device=DEV).manual_seed(m + n)
    w = (torch.randn(n, k, device=DEV, generator=g) * 0.02).to(BF)
    x = torch.randn(m, k, device=DEV, generator=g).to(BF)
    new, old = torch.empty(m, n, device=DEV, dtype=BF), torch.empty(m, n, device=DEV)
    status = torch.zeros(1, device=DEV, dtype=torch.int32)
    a = lib.GemmSmallMArgs(w=lib.ptr(w), x=lib.ptr(x), y=lib.ptr(new), status=lib.ptr(status), m=m, n=n, k=k)
    lib.check(so.tfb_gemm_rows(C.byref(a), lib.stream()), "tfb_gemm_rows")
    xf = x.float()
    for t in range(m):
        a = lib.GemvF32Args(w=lib.ptr(w), x=lib.ptr(xf[t]), y=lib.ptr(old[t]), n=n, k=k, eps=1e-6, prologue=lib.NORM_NONE, epilogue=0)
        lib.check(so.tfb_gemv_f32(C.byref(a), lib.stream()), "tfb_gemv_f32")
    assert int(status) == 0 and torch.equal(old, old.to(BF).float())
    _no_worse(f"projection {m} x {n} x {k}", new, old.to(BF), x.double() @ w.double().t())
