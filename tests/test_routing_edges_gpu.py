"""Routing where the logits or indices are not what a healthy model gives: nothing is read or written out of range, and the
tokens that are healthy get what they get without the others."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
BF, DEV = torch.bfloat16, "cuda:0"
NAN, INF = float("nan"), float("inf")
E, K, H, I, T = 16, 4, 256, 256, 21


@pytest.fixture(scope="module")
def so():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tilefoundry_b200 import lib
    return lib.load()


# all NaN, one number left, -infinity in the rest, +infinity (its softmax over all experts is NaN), fewer numbers than selections
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("fill,at", [(NAN, {}), (NAN, {5: 1.0}), (-INF, {5: 1.0}), (0.0, {3: INF}), (NAN, {0: -INF, 9: 2.0, 11: 2.0})])
def test_selection_names_different_experts_whatever_the_logits(so, mode, fill, at):
    from tilefoundry_b200 import lib
    for experts, top_k in ((E, K), (E, E), (200, 32)):
        logits = torch.full((experts,), fill)
        for i, v in at.items():
            logits[i] = v
        idx, weight = torch.full((top_k,), -7, dtype=torch.int64, device=DEV), torch.empty(top_k, device=DEV)
        on_gpu = logits.to(DEV)
        lib.check(so.tfb_router_select(None, lib.ptr(on_gpu), lib.ptr(idx), None, lib.ptr(weight), experts, top_k, mode, 0, lib.stream()),
                  "tfb_router_select")
        got = idx.tolist()
        assert len(set(got)) == top_k and all(0 <= e < experts for e in got)
        if INF not in at.values() or mode == 0:               # the numbers first, by value, then index
            first = sorted((e for e in range(experts) if logits[e] == logits[e]), key=lambda e: (-float(logits[e]), e))
            assert got[: len(first)] == first[:top_k]


def _block(so, x, indices=None):
    from tilefoundry_b200 import lib
    g = torch.Generator(device=DEV).manual_seed(3)
    weight = lambda *s: (torch.randn(*s, device=DEV, generator=g) * 0.06).to(BF)
    empty = lambda *s, dtype=torch.float32: torch.zeros(*s, device=DEV, dtype=dtype)
    i32, i64 = torch.int32, torch.int64
    keep = dict(w_router=weight(E, H), w_shared_scale=weight(1, H), w_gate=weight(E, I, H), w_up=weight(E, I, H), w_down=weight(E, H, I),
                w_shared_gate=weight(I, H), w_shared_up=weight(I, H), w_shared_down=weight(H, I), logits=empty(T, E + 1),
                indices=empty(T, K, dtype=i64), weights=empty(T, K), shared_gate=empty(T), out=empty(T, H), status=empty(1, dtype=i32),
                x_bf16=empty(T, H, dtype=BF), inner=empty(T, K + 1, I, dtype=BF), y=empty(T, K + 1, H, dtype=BF),
                counts=empty(2 * (E + 1) + 1, dtype=i32), lists=torch.full((E + 1, T), -1, dtype=i32, device=DEV), x=x)
    at = {n: lib.ptr(t) for n, t in keep.items()}
    pick = lambda *names: {n: at[n] for n in names}
    route = lib.MoeRouteArgs(tokens=T, hidden=H, experts=E, top_k=K, mode=1, pdl=0,
                             **pick("x", "w_router", "w_shared_scale", "logits", "indices", "weights", "shared_gate"))
    lib.check(so.tfb_moe_batch_route(C.byref(route), lib.stream()), "tfb_moe_batch_route")
    if indices is not None:
        keep["indices"].copy_(indices)
    block = lib.MoeBatchArgs(residual=None, tokens=T, hidden=H, inter=I, experts=E, top_k=K, pdl=0,
                             **pick("x", "indices", "weights", "shared_gate", "w_gate", "w_up", "w_down", "w_shared_gate", "w_shared_up",
                                    "w_shared_down", "out", "status", "x_bf16", "inner", "y", "counts", "lists"))
    lib.check(so.tfb_moe_batch(C.byref(block), lib.stream()), "tfb_moe_batch")
    assert int(keep["status"]) == 0
    return keep


def _tokens():
    return torch.randn(T, H, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5))


@pytest.mark.parametrize("bad", [NAN, INF])
def test_a_token_that_is_not_finite_leaves_the_others_alone(so, bad):
    clean = _block(so, _tokens())
    x = _tokens()
    x[7] = bad
    got = _block(so, x)
    others = [t for t in range(T) if t != 7]
    for name in ("indices", "weights", "out"):
        assert torch.equal(got[name][others], clean[name][others]), name
    assert len(set(got["indices"][7].tolist())) == K and int(got["indices"].min()) >= 0 and int(got["indices"].max()) < E
    assert not torch.isfinite(got["out"][7]).any()


@pytest.mark.parametrize("index", [-1, E, E + 1, 0x7fffffff, 1 << 40, -(1 << 63)])
def test_an_index_that_names_no_expert_is_on_no_list(so, index):
    clean = _block(so, _tokens())
    indices = clean["indices"].clone()
    indices[2, 1] = indices[T - 1, K - 1] = index
    got = _block(so, _tokens(), indices=indices)
    others = [t for t in range(T) if t not in (2, T - 1)]
    assert torch.equal(got["out"][others], clean["out"][others])
    counts = [int((indices == e).sum()) for e in range(E)]
    assert got["counts"][:E].tolist() == counts and int(got["counts"][E]) == T
    entries = [[int(t) << 8 | int(s) for t, s in (indices == e).nonzero().tolist()] for e in range(E)] + [[t << 8 | K for t in range(T)]]
    for e, want in enumerate(entries):
        assert got["lists"][e].tolist() == want + [-1] * (T - len(want)), f"list {e}"


def test_an_expert_named_more_often_than_there_are_tokens_stays_on_its_own_list(so):
    got = _block(so, _tokens(), indices=torch.full((T, K), 4, device=DEV))
    assert int(got["counts"][4]) == T
    assert got["lists"][4].tolist() == [a // K << 8 | a % K for a in range(T)]
    for e in range(E):
        if e != 4:
            assert got["lists"][e].tolist() == [-1] * T
    assert got["lists"][E].tolist() == [t << 8 | K for t in range(T)]
