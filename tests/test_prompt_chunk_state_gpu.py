"""What a chunked prompt leaves behind: all of the state and outputs that the token-by-token walk leaves."""
import pytest
import torch

from tests.helpers import assert_close_at_scale
from tilefoundry_b200.authored import minicpm3_4b as mc
from tilefoundry_b200.authored import qwen3_1_7b as q
from tilefoundry_b200.authored import qwen3_5_35b_a3b as q35
from tilefoundry_b200.authored.weights import random_weights
from tilefoundry_b200.runtime import DictResource

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qwen35():
    """``session(n_prompt) -> (session, prompt)`` over one set of weights whose rounding flips no expert that counts."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tilefoundry_b200 import lib
    from tilefoundry_b200.engine.qwen3_5 import Qwen35Session
    lib.load()
    cfg = q35.QWEN3_5_TINY
    w = random_weights(q35.build(cfg), seed=9, std=0.05, overrides=q35.weight_overrides)
    for name, t in w.items():
        leaf = name.rsplit(".", 1)[-1]
        t *= 0.02 if leaf in ("w_o", "w_out", "w_down", "w_shared_down") else 3.0 if leaf == "w_router" else 1.0
    res = DictResource({k: v.to("cuda:0") for k, v in w.items()})

    def session(n_prompt):
        sess = Qwen35Session(cfg, res, max_ctx=128, device="cuda:0", keep_logits=True)
        return sess, torch.randint(0, cfg.vocab_size, (n_prompt,), generator=torch.Generator().manual_seed(n_prompt))
    return session


# chunks of 2 and 3 reach back into the window before them; odd and even lengths and starts swap the two windows' buffers
@pytest.mark.parametrize("pieces", [(2,), (3,), (4,), (17,), (40,), (2, 2), (2, 3), (3, 2), (5, 4), (16, 21)])
def test_chunks_leave_both_convolution_windows(qwen35, pieces):
    (walk, prompt), (pre, _) = qwen35(sum(pieces) + 1), qwen35(sum(pieces) + 1)
    walk.reset(prompt), pre.reset(prompt)
    for _ in range(sum(pieces)):
        walk.step()
    for n in pieces:
        pre.prefill(n)
    pre._prefill.check_status()
    assert int(pre.pos) == int(walk.pos) == sum(pieces)
    assert len(pre.state_tensors()) == len(walk.state_tensors()) > 0
    for i, (got, want) in enumerate(zip(pre.state_tensors(), walk.state_tensors())):
        assert got.shape == want.shape
        for part, (a, b) in enumerate(zip(got, want)):      # a window, or a head's state, at its own scale
            assert_close_at_scale(a, b, f"state tensor {i} part {part}")


@pytest.mark.parametrize("use_graph", [False, True])
def test_steps_inside_a_prompt_leave_their_logits_and_picks(qwen35, use_graph):
    """``run`` takes the positions of a part of a prompt as steps: a caller who scores a prompt piece by piece reads each
    piece's last logits and pick, and nothing waits for the device."""
    (walk, prompt), (sess, _) = qwen35(10), qwen35(10)
    walk.reset(prompt)
    sess.generate(prompt.flip(0), 1)                     # another request's logits and pick lie there
    sess.reset(prompt)
    for steps in (5, 3, 2):                              # inside the prompt, and its end
        for _ in range(steps):
            walk.step()
        torch.cuda.set_sync_debug_mode("error")          # (a device read inside run raises)
        try:
            sess.run(steps, use_graph)
        finally:
            torch.cuda.set_sync_debug_mode("default")
        assert torch.equal(sess.logits, walk.logits) and int(sess.picked) == int(walk.picked) and int(sess.pos) == int(walk.pos)
    for got, want in zip(sess.state_tensors(), walk.state_tensors()):
        assert torch.equal(got, want)


@pytest.mark.parametrize("steps", [10, 11, 25])
def test_steps_past_a_prompt_go_on_as_generate_does(qwen35, steps):
    (gen, prompt), (sess, _) = qwen35(10), qwen35(10)
    want = gen.generate(prompt, steps - 9).tokens
    sess.reset(prompt)
    start = sess.snapshot()
    for _ in range(2):                                   # (and again from the start)
        sess.run(steps)
        assert sess.tokens[10: steps + 1].tolist() == want and int(sess.pos) == steps and int(sess.picked) == want[-1]
        assert torch.equal(sess.logits, gen.logits)
        for got, other in zip(sess.state_tensors(), gen.state_tensors()):
            assert torch.equal(got, other)
        sess.restore(start)
    sess.run(4)                                          # not at the start any more: no chunk may begin there
    sess.run(12)
    sess.check_prompt()
    assert int(sess.pos) == 16


def _chunked_session(model, qwen35):
    if model == "qwen3.5":
        return qwen35(8)
    from tilefoundry_b200.engine.minicpm3 import MiniCPM3Session
    from tilefoundry_b200.engine.qwen3 import Qwen3Session
    mod, cfg, cls = (q, q.QWEN3_SMALL, Qwen3Session) if model == "qwen3" else (mc, mc.MINICPM3_TINY, MiniCPM3Session)
    w = mod.tie_head(random_weights(mod.build(cfg), seed=7, std=0.02))
    sess = cls(cfg, DictResource({k: v.to("cuda:0") for k, v in w.items()}), max_ctx=64, device="cuda:0")
    return sess, torch.randint(0, cfg.vocab_size, (8,), generator=torch.Generator().manual_seed(8))


@pytest.mark.parametrize("model", ["qwen3", "minicpm3", "qwen3.5"])
def test_a_given_up_wait_of_a_chunk_is_told_once(model, qwen35):
    """The status word as a kernel that gave up leaves it (set from the host): the next call that waits for the stream raises."""
    sess, prompt = _chunked_session(model, qwen35)
    token_in, token_out = (torch.zeros(1, dtype=torch.int64).pin_memory() for _ in range(2))
    calls = {"step_host": lambda: sess.step_host(6, token_in, token_out), "generate_host": lambda: sess.generate_host(6, 1, token_in),
             "check_prompt": sess.check_prompt}
    for call in calls.values():
        sess.reset(prompt)
        sess.prefill(6)
        sess._prefill.status.fill_(2)
        with pytest.raises(RuntimeError, match="bounded wait"):
            call()
        call()                                           # told once
    assert not sess.prompt_unchecked
    sess.reset(prompt)
    sess.prefill(6)
    sess._prefill.status.fill_(2)
    with pytest.raises(RuntimeError, match="bounded wait"):
        sess.generate(prompt, 2, prefill=True)
    assert len(sess.generate(prompt, 2, prefill=True).tokens) == 2


@pytest.mark.parametrize("model", ["qwen3", "minicpm3", "qwen3.5"])
def test_generate_is_asked_for_chunks_or_a_walk(model, qwen35):
    """``prefill`` of ``generate`` on every session that has chunks; without it each keeps its own default."""
    sess, prompt = _chunked_session(model, qwen35)
    walked = sess.generate(prompt, 3, prefill=False)
    assert sess._prefill is None and walked.prompt_steps == 8
    assert sess.generate(prompt, 3, True, None if model == "qwen3.5" else False).prompt_steps == 8      # (the fourth argument as before)
    chunked = sess.generate(prompt, 3, prefill=True)
    assert sess._prefill is not None and len(chunked.tokens) == len(walked.tokens) == 3 and int(sess.pos) == 10
