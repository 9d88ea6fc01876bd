"""The nucleus draw where logits are infinite or not numbers."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import sampling

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _draw(logits, temperature, top_p, seed, step):
    from tilefoundry_b200 import lib
    i32, i64 = torch.int32, torch.int64
    keep = dict(logits=logits, pos=torch.tensor([step + 1], dtype=i32, device="cuda"), prev_pos=torch.tensor([step], dtype=i32, device="cuda"),
                tokens=torch.full((step + 4,), -1, dtype=i64, device="cuda"), picked=torch.full((1,), -1, dtype=i64, device="cuda"),
                hist=torch.zeros(65536 + 128, dtype=i32, device="cuda"))
    a = lib.SampleTopPArgs(**{n: lib.ptr(t) for n, t in keep.items()}, vocab=logits.numel(), n_prompt=0, n_eos=0, pdl=0,
                           temperature=temperature, top_p=top_p, seed=seed)
    for _ in range(2):                                   # (the second call finds what the first one left of its scratch)
        lib.check(lib.load().tfb_sample_top_p(C.byref(a), lib.stream()), "tfb_sample_top_p")
    assert keep["tokens"].tolist()[step + 1] == int(keep["picked"]) and not keep["hist"][:65536].any()
    return int(keep["picked"])


# one infinite logit, several (in one warp, in several CTAs), an overflow of logit / temperature, and the last of a ragged end
@pytest.mark.parametrize("vocab", [33, 1000, 151936])
@pytest.mark.parametrize("temperature", [0.8, 1e-6])
def test_the_pick_among_infinite_logits_is_the_lowest_index(vocab, temperature):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator(device="cuda").manual_seed(vocab)
    base = (torch.randn(vocab, device="cuda", generator=g) * 3).to(torch.bfloat16)
    for where in ([0], [vocab - 1], [vocab // 2, vocab // 2 + 1], [vocab - 1, vocab // 3, vocab // 2]):
        for value in (INF, 3e38):                        # (3e38 / temperature overflows)
            logits = base.clone()
            logits[where] = value
            assert _draw(logits, temperature, 0.9, 5, 7) == min(where), (where, value)


@pytest.mark.parametrize("vocab", [33, 151936])
def test_minus_infinity_and_nan_are_not_drawn_while_there_is_a_number(vocab):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator(device="cuda").manual_seed(vocab)
    base = (torch.randn(vocab, device="cuda", generator=g) * 3).to(torch.bfloat16)
    half = torch.arange(vocab, device="cuda") % 2 == 0
    for step in range(4):
        masked = torch.where(half, torch.full_like(base, -INF), base)
        assert _draw(masked, 0.8, 0.9, 11, step) == sampling.sample_top_p(masked.float().cpu().numpy(), 0.8, 0.9, 11, step)
        broken = torch.where(half, torch.full_like(base, NAN), base)      # (no nucleus is defined: a draw from all the numbers)
        scores = sampling.gumbel_scores(broken.float().cpu().numpy(), 0.8, 11, step)
        assert _draw(broken, 0.8, 0.9, 11, step) == int(np.nanargmax(scores))
    assert _draw(torch.full_like(base, -INF), 0.8, 0.9, 11, 0) == 0
