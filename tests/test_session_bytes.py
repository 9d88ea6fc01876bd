"""Byte counts that sessions give out, from the layers a session holds (no device: the counting methods only)."""
import pytest

from tests.test_packed_models import MODELS
from tilefoundry_b200.authored import qwen3_1_7b as q
from tilefoundry_b200.authored.weights import random_weights
from tilefoundry_b200.engine import packed, packed_models
from tilefoundry_b200.engine.granite import GraniteSession
from tilefoundry_b200.engine.minicpm3 import MiniCPM3Session
from tilefoundry_b200.engine.qwen3 import Qwen3Session
from tilefoundry_b200.engine.qwen3_5 import Qwen35Session
from tilefoundry_b200.engine.qwen3_batch import Qwen3BatchSession
from tilefoundry_b200.runtime import DictResource


def _qwen3(cls):
    cfg = q.QWEN3_SMALL
    return cls, cfg, packed.pack(cfg, DictResource(q.tie_head(random_weights(q.build(cfg), seed=1))))


def _other(model, cls):
    cfg, w = MODELS[model]()
    return cls, cfg, packed_models.pack(model, cfg, DictResource(w))


SESSIONS = {"qwen3": lambda: _qwen3(Qwen3Session), "qwen3 batch": lambda: _qwen3(Qwen3BatchSession),
            "minicpm3": lambda: _other("minicpm3_4b", MiniCPM3Session), "granite": lambda: _other("granite_4_0_h_small", GraniteSession),
            "qwen3.5": lambda: _other("qwen3_5_35b_a3b", Qwen35Session)}


@pytest.mark.parametrize("name", SESSIONS)
def test_every_byte_count_is_given(name):
    cls, cfg, weights = SESSIONS[name]()
    sess = object.__new__(cls)
    sess.cfg, sess.world, sess.cache, sess.batch = cfg, 1, "latent", 2
    kinds = getattr(cfg, "layer_types", [None] * len(weights.layers))
    sess.layers = [{**layer, "kind": kind} for layer, kind in zip(weights.layers, kinds)]
    for layer in sess.layers:
        if "w_gate_up" in layer:                          # (sessions hold the halves too)
            layer["w_gate"], layer["w_up"] = layer["w_gate_up"].chunk(2)
    sess.w_head = weights.root["w_embed"] if "w_embed" in weights.root else None       # a tied head
    for n, t in weights.root.items():
        if t is not None:
            setattr(sess, {"table": "table_w"}.get(n, n), t)
    counts = [n for n in ("weight_bytes", "kv_bytes_per_position", "state_bytes") if hasattr(cls, n)]
    assert "weight_bytes" in counts
    for n in counts:
        assert isinstance(getattr(sess, n)(), int) and getattr(sess, n)() > 0, n
    if name == "granite":
        recurrent = sum(k == "linear_attention" for k in cfg.layer_types)
        assert sess.state_bytes() == 8 * recurrent * cfg.mamba_n_heads * cfg.mamba_d_head * cfg.mamba_d_state
