"""Edges of the decode-step and prompt-chunk kernels' variants: remainders, unaligned results, ties and infinities in the
expert selection, the first token picked by the chunk itself."""
import ctypes as C

import pytest
import torch

from tests.helpers import assert_ulps
from tilefoundry_b200.authored import qwen3_1_7b as q
from tilefoundry_b200.authored.weights import random_weights
from tilefoundry_b200.runtime import DictResource

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tilefoundry_b200 import lib
    lib.load()
    return torch.device("cuda:0")


# 4096 rows on: the persistent form; a row more than whole tiles, K of one batch and of a ragged last batch
@pytest.mark.parametrize("n,k", [(4095, 512), (4096, 256), (4097, 1280), (12352, 2048), (9217, 8192)])
def test_f32_input_projection_matches_f64(dev, n, k):
    from tilefoundry_b200 import lib
    g = torch.Generator(device=dev).manual_seed(n + k)
    w = (torch.randn(n, k, device=dev, generator=g) * k ** -0.5).to(BF)
    x = torch.randn(k, device=dev, generator=g)
    gain = 1 + 0.1 * torch.randn(k, device=dev, generator=g)
    y = torch.empty(n, device=dev)
    a = lib.GemvF32Args(w=lib.ptr(w), x=lib.ptr(x), gamma=lib.ptr(gain), y=lib.ptr(y), n=n, k=k, eps=1e-6,
                        prologue=lib.NORM_F32GAIN, epilogue=0)
    lib.check(lib.load().tfb_gemv_f32(C.byref(a), lib.stream()), "tfb_gemv_f32")
    normed = (x * torch.rsqrt(x.square().mean() + 1e-6) * gain).to(BF)
    want = (w.double() @ normed.double()).float()
    # a step of bf16 for the result's rounding, and the roundings of the normalised vector that another order of its sum of
    # squares moves (at most one in a few hundred elements, by a step of bf16 each)
    assert (y - want).abs().max().item() < 2 ** -8 * want.abs().max().item() + 2 ** -8


# results that start between 8-byte boundaries: stored one at a time
@pytest.mark.parametrize("m,n,k", [(5, 64, 128), (32, 2048, 2048), (200, 512, 256)])
def test_projection_into_an_odd_address(dev, m, n, k):
    from tilefoundry_b200 import lib
    g = torch.Generator(device=dev).manual_seed(m)
    w = (torch.randn(n, k, device=dev, generator=g) * k ** -0.5).to(BF)
    x = torch.randn(m, k, device=dev, generator=g).to(BF)
    y = torch.empty(m * n + 1, device=dev, dtype=BF)
    status = torch.zeros(1, device=dev, dtype=torch.int32)
    a = lib.GemmSmallMArgs(w=lib.ptr(w), x=lib.ptr(x), y=y.data_ptr() + 2, status=lib.ptr(status), m=m, n=n, k=k)
    call = lib.load().tfb_gemm_small_m if m <= 32 else lib.load().tfb_gemm_rows
    lib.check(call(C.byref(a), lib.stream()), "projection")
    assert int(status) == 0
    assert_ulps(y[1:].view(m, n).cpu(), (x.double() @ w.double().t()).to(BF).cpu(), 1, "y")


# token tiles of 128 and 256, splits of two, three (uneven K steps) and four
@pytest.mark.parametrize("m", [128, 129, 193, 256, 509])
@pytest.mark.parametrize("n,k", [(2048, 6144), (2304, 512), (2432, 512), (2560, 6400)])
def test_token_tiles_and_splits(dev, m, n, k):
    from tilefoundry_b200 import lib
    g = torch.Generator(device=dev).manual_seed(m + n)
    w = (torch.randn(n, k, device=dev, generator=g) * k ** -0.5).to(BF)
    x, res = (torch.randn(m, c, device=dev, generator=g).to(BF) for c in (k, n))
    y = torch.empty(m, n, device=dev, dtype=BF)
    status = torch.zeros(1, device=dev, dtype=torch.int32)
    a = lib.GemmSmallMArgs(w=lib.ptr(w), x=lib.ptr(x), y=lib.ptr(y), residual=lib.ptr(res), status=lib.ptr(status), m=m, n=n, k=k)
    lib.check(lib.load().tfb_gemm_rows(C.byref(a), lib.stream()), "tfb_gemm_rows")
    assert int(status) == 0
    # the product's rounding may fall on either side (one step of the product's own scale, up to 2^-7 of 4), then the sum's
    prod = x.double() @ w.double().t()
    want = res.double() + prod.to(BF).double()
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -7 * prod.abs() + 1e-6).all()


# either side of the lines between split counts: clusters of four and three, two splits on a shared SM, halves of 128 tokens
@pytest.mark.parametrize("m,n,k", [(129, 4224, 512), (129, 4352, 512), (200, 5632, 320), (200, 5760, 320), (192, 2304, 512), (193, 2304, 512),
                                   (33, 9472, 256), (128, 9600, 256), (64, 4864, 512), (100, 2304, 1024), (32, 4736, 512), (500, 2176, 320)])
def test_lines_between_split_counts(dev, m, n, k):
    test_token_tiles_and_splits(dev, m, n, k)


@pytest.mark.parametrize("experts,top_k", [(5, 5), (72, 10), (128, 32), (256, 8)])
def test_selection_orders_ties_zeros_and_infinities(dev, experts, top_k):
    from tilefoundry_b200 import lib
    g = torch.Generator().manual_seed(experts)
    rows = [torch.randn(experts, generator=g), torch.zeros(experts), torch.where(torch.arange(experts) % 2 == 0, 0.0, -0.0),
            (torch.randn(experts, generator=g) * 2).round(), -torch.rand(experts, generator=g)]
    rows[3][: experts // 2] = -float("inf")
    for logits in rows:
        idx = torch.empty(top_k, dtype=torch.int64, device=dev)
        weight = torch.empty(top_k, device=dev)
        on_gpu = logits.to(dev)
        lib.check(lib.load().tfb_router_select(None, lib.ptr(on_gpu), lib.ptr(idx), None, lib.ptr(weight), experts, top_k, 0, 0,
                                               lib.stream()), "tfb_router_select")
        order = torch.sort(logits, descending=True, stable=True).indices[:top_k]
        n = min(int(torch.isfinite(logits).sum()), top_k)
        assert idx.cpu()[:n].tolist() == order[:n].tolist()
        torch.testing.assert_close(weight.cpu()[:n], torch.softmax(logits[order], 0)[:n], rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("n_prompt", [2, 3, 40])
def test_first_token_of_a_chunked_prompt_is_drawn_and_ended_as_by_a_step(dev, n_prompt):
    from oracle import sampling
    from tilefoundry_b200.engine.qwen3 import Qwen3Session
    cfg = q.QWEN3_SMALL
    res = DictResource({k: v.to(dev) for k, v in q.tie_head(random_weights(q.build(cfg), seed=7, std=0.02)).items()})
    prompt = torch.randint(0, cfg.vocab_size, (n_prompt,), generator=torch.Generator().manual_seed(n_prompt))
    for options in ({}, {"temperature": 0.8, "seed": 42}, {"temperature": 0.8, "seed": 42, "top_p": 0.6}):
        sess = Qwen3Session(cfg, res, max_ctx=64, device=dev, keep_logits=True, **options)
        first = sess.generate(prompt, 1, prefill=True).tokens
        logits = sess.logits.float().cpu().numpy()
        want = (int(logits.argmax()) if not options else sampling.sample_top_p(logits, 0.8, 0.6, 42, n_prompt - 1) if "top_p" in options
                else sampling.sample(logits, 0.8, 42, n_prompt - 1))
        assert first == [want] and int(sess.pos) == n_prompt and int(sess.picked) == want
        assert sess.generate(prompt, 5, prefill=True, eos=[want]).tokens == []
        assert sess.generate(prompt, 0, prefill=True, eos=[]).tokens == []
        assert int(sess.pos) == n_prompt - 1
