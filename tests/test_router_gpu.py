"""Routers with several tokens a block, and the sort of their choices by expert, at the sizes where they change their form: more than 64
tokens, last blocks of one to three tokens, odd numbers of experts, many pairs a warp, more experts than shared memory has
counts for 32 warps."""
import pytest
import torch

import kernel_utils as K
from atoma_infer_b200.csrc import ops as O

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
@pytest.mark.parametrize("T", [64, 65, 67, 130])
@pytest.mark.parametrize("H,E,top", [(136, 5, 2), (100, 37, 4), (97, 16, 3), (512, 130, 8), (64, 3, 3)])
def test_choices_and_weights(rts, dtype, kind, T, H, E, top):
    rt = rts[dtype]
    h, w, more = inputs(rt, T, H, E)
    ids, wts = route(rt, kind, h, w, more, top)
    ids = ids.long()
    z = h.double() @ w.double().T
    if kind == "sigmoid":
        score = torch.sigmoid(z) + more.double()
        want = torch.gather(torch.sigmoid(z), 1, ids)
    else:
        score = z + more.double()
        p = torch.softmax(score, -1)
        want = torch.gather(p, 1, ids)
        want = want / want.sum(-1, keepdim=True)
    assert bool((ids.sort(1).values.diff(dim=1) > 0).all())
    # logits of up to 512 products, float32: a few 1e-6; neighbours closer than that may change places
    assert torch.allclose(torch.gather(score, 1, ids), score.topk(top, -1).values, atol=1e-5, rtol=0)
    assert torch.allclose(wts.double(), want, atol=1e-5, rtol=0)


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


def sort(rt, ids, T, top, E):
    dev = ids.to(rt.device)
    offsets = torch.full((E + 1,), -1, dtype=torch.int32, device=rt.device)
    order, place = (torch.full((T * top,), -1, dtype=torch.int32, device=rt.device) for _ in range(2))
    rt.ops._check(rt.ops._mixers().moe_sort(O._p(dev), O._p(offsets), O._p(order), O._p(place), O._p(meta(rt, T)), top, E, rt.ops._stream()), "moe_sort")
    return offsets.cpu().long(), order.cpu().long(), place.cpu().long()


@pytest.mark.parametrize("top", [1, 3])
@pytest.mark.parametrize("T", [1, 31, 1025, 3001, 4097, 9001])
@pytest.mark.parametrize("E", [1, 16, 37, 400, 1000])
@pytest.mark.parametrize("skewed", [False, True])
def test_sort_by_expert(rts, top, T, E, skewed):
    n = T * top
    x = torch.rand(n, generator=torch.Generator().manual_seed(T + E))
    ids = ((x ** 6 if skewed else x) * E).int().clamp_(max=E - 1)
    offsets, order, place = sort(rts["bfloat16"], ids, T, top, E)
    want = torch.argsort(ids.long(), stable=True)
    assert torch.equal(order, want) and torch.equal(place[want], torch.arange(n))
    assert torch.equal(offsets, torch.cat([torch.zeros(1, dtype=torch.int64), torch.bincount(ids.long(), minlength=E).cumsum(0)]))


def test_sort_leaves_out_what_names_no_expert(rts):
    T, E = 3001, 37
    ids = torch.randint(-2, E + 4, (T,), generator=torch.Generator().manual_seed(0), dtype=torch.int32)
    ids[::500] = 1 << 30
    offsets, order, place = sort(rts["bfloat16"], ids, T, 1, E)
    real = ((ids >= 0) & (ids < E)).nonzero()[:, 0]
    want = real[torch.argsort(ids[real].long(), stable=True)]
    assert torch.equal(order[:len(real)], want) and bool((order[len(real):] == -1).all()) and int(offsets[-1]) == len(real)
    assert torch.equal(place[want], torch.arange(len(real))) and int((place >= 0).sum()) == len(real)
