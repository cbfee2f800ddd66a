"""Routers with several tokens a block: the same choice and weights wherever a token stands."""
import pytest
import torch

import kernel_utils as K

pytestmark = pytest.mark.gpu
KINDS = ["softmax", "over_chosen", "sigmoid"]


@pytest.fixture(scope="module")
def rts():
    from atoma_infer_b200.engine.runtime import make_runtime

    return {d: make_runtime(d, "cuda:0") for d in ("float32", "bfloat16")}


def meta(rt, T):
    return K.make_context(rt, [(0, T)], 16, [[1] * (-(-T // 16))])[0].meta


def route(rt, kind, h, w, more, top):
    """more: the logits' bias, or the sigmoid router's correction."""
    ids, wts = torch.full((h.shape[0], top), -1, dtype=torch.int32, device=rt.device), torch.full((h.shape[0], top), float("nan"), device=rt.device)
    if kind == "sigmoid":
        rt.ops.moe_route_sigmoid(h, w, more, ids, wts, meta(rt, h.shape[0]))
    else:
        rt.ops.moe_route(h, w, ids, wts, meta(rt, h.shape[0]), bias=more, over_chosen=kind == "over_chosen")
    return ids, wts


def inputs(rt, T, H, E):
    g = torch.Generator().manual_seed(H + E)
    return (torch.randn(T, H, generator=g).to(rt.dtype).to(rt.device), (torch.randn(E, H, generator=g) * 0.2).to(rt.device),
            (torch.randn(E, generator=g) * 0.5).to(rt.device))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("H", [100, 136, 97])  # (bfloat16 rows of 100: every second one starts on 8 bytes, not 16)
def test_a_token_is_routed_alike_wherever_it_stands(rts, dtype, kind, H):
    rt = rts[dtype]
    h, w, more = inputs(rt, 150, H, 37)
    ids, wts = route(rt, kind, h, w, more, 4)
    for first, n in ((0, 7), (1, 1), (2, 1), (3, 64), (83, 67)):
        some = route(rt, kind, h[first:first + n].clone(), w, more, 4)
        assert torch.equal(some[0], ids[first:first + n]) and torch.equal(some[1], wts[first:first + n])
