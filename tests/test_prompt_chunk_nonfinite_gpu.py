"""Values that are not finite, next to a prompt chunk and inside it: what a token must not see does not reach it."""
import pytest
import torch

from tests.helpers import assert_close_at_scale
from tilefoundry_b200.authored import minicpm3_4b as mc
from tilefoundry_b200.authored import qwen3_1_7b as q
from tilefoundry_b200.authored import qwen3_5_35b_a3b as q35
from tilefoundry_b200.authored.weights import random_weights
from tilefoundry_b200.runtime import DictResource

pytestmark = pytest.mark.gpu
DEV, MAX_CTX = "cuda:0", 256


def _qwen3():
    from tilefoundry_b200.engine.qwen3 import Qwen3Session
    return Qwen3Session, q.QWEN3_SMALL, q.tie_head(random_weights(q.build(q.QWEN3_SMALL), seed=7, std=0.02)), "w_embed"


def _minicpm3():
    from tilefoundry_b200.engine.minicpm3 import MiniCPM3Session
    return MiniCPM3Session, mc.MINICPM3_TINY, mc.tie_head(random_weights(mc.build(mc.MINICPM3_TINY), seed=5, std=0.02)), "w_embed"


def _qwen35():
    from tilefoundry_b200.engine.qwen3_5 import Qwen35Session
    w = random_weights(q35.build(q35.QWEN3_5_TINY), seed=9, std=0.05, overrides=q35.weight_overrides)
    for name, t in w.items():                            # small branches and a decided router: rounding flips no expert that counts
        leaf = name.rsplit(".", 1)[-1]
        t *= 0.02 if leaf in ("w_o", "w_out", "w_down", "w_shared_down") else 3.0 if leaf == "w_router" else 1.0
    return Qwen35Session, q35.QWEN3_5_TINY, w, "table"


@pytest.fixture(scope="module", params=["qwen3", "minicpm3", "qwen3.5"])
def make(request):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tilefoundry_b200 import lib
    lib.load()
    cls, cfg, w, embed = {"qwen3": _qwen3, "minicpm3": _minicpm3, "qwen3.5": _qwen35}[request.param]()

    def session(bad=None):
        ours = {k: v.to(DEV) for k, v in w.items()}
        if bad is not None:
            ours[embed] = ours[embed].clone()
            ours[embed][bad] = float("nan")
        return cls(cfg, DictResource(ours), max_ctx=MAX_CTX, device=DEV, keep_logits=True)
    session.vocab = cfg.vocab_size
    return session


def _pools(sess):
    return [(f"layer {i} {n}", layer[n]) for i, layer in enumerate(sess.layers) for n in ("k_pool", "v_pool") if layer.get(n) is not None]


def _prompt(make, n):
    return torch.randint(0, make.vocab - 1, (n,), generator=torch.Generator().manual_seed(n))


@pytest.mark.parametrize("stale", [float("nan"), float("inf")])
@pytest.mark.parametrize("n_prompt,piece", [(3, 256), (63, 256), (64, 256), (65, 256), (130, 256), (200, 256), (200, 70)])
def test_stale_rows_past_the_prompt_are_not_seen(make, n_prompt, piece, stale):
    """A cache that was never initialised, or holds what an earlier request overflowed to."""
    sess, prompt = make(), _prompt(make, n_prompt)
    sess.generate(prompt, 1, prefill=True)
    sess._prefill.chunk = piece
    results = []
    for fill in (0.0, stale):
        for _, pool in _pools(sess):
            pool.fill_(fill)
        sess.generate(prompt, 1, prefill=True)
        results.append([sess.logits.clone()] + [pool.view(-1, *pool.shape[2:])[:n_prompt].clone() for _, pool in _pools(sess)])
    assert torch.isfinite(results[0][0]).all()
    for clean, got in zip(*results):
        assert torch.equal(clean, got)


# the bad token in the first, a middle and the last place of query tiles of 64 and 128 tokens, in one chunk and in two
@pytest.mark.parametrize("n_prompt,bad,piece", [(5, 2, 256), (64, 63, 256), (100, 1, 256), (150, 70, 256), (200, 128, 256), (200, 127, 256), (200, 150, 120)])
def test_a_token_that_is_not_finite_reaches_no_earlier_one(make, n_prompt, bad, piece):
    walk, pre = make(make.vocab - 1), make(make.vocab - 1)
    prompt = _prompt(make, n_prompt)
    prompt[bad] = make.vocab - 1
    walk.reset(prompt)
    for _ in range(n_prompt):
        walk.step()
    pre.reset(prompt)
    pre._chunks().chunk = piece
    pre.prefill(n_prompt)
    pre.check_prompt()
    for (name, a), (_, b) in zip(_pools(pre), _pools(walk)):
        a, b = (x.view(-1, *x.shape[2:])[:n_prompt] for x in (a, b))
        assert torch.isfinite(b[:bad]).all() and torch.equal(torch.isfinite(a), torch.isfinite(b)), name
        assert_close_at_scale(a[:bad], b[:bad], name)
        after = torch.isfinite(b[bad:])
        if after.any():
            assert_close_at_scale(a[bad:][after], b[bad:][after], f"{name}, from the token on")
