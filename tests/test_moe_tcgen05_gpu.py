"""Routed experts' linears on tcgen05: stretches of no, one, 15 to 17, 255 to 257 and 600 rows, results that are no multiple of a tile's 64 or
128 rows, depths that are no multiple of 64, with the shared expert in the same launches and without it."""
import pytest
import torch

import kernel_utils as K

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from atoma_infer_b200.engine.runtime import make_runtime

    return make_runtime("bfloat16", "cuda:0")


@pytest.mark.parametrize("H,F,Fs", [(136, 72, 40), (256, 128, 0), (520, 200, 264), (64, 8, 8)])
@pytest.mark.parametrize("counts,top", [([0, 1, 15, 16, 17, 0, 255, 256, 257, 600, 3], 2), ([128], 1), ([0, 0, 130, 0], 1), ([300] * 40, 3)])
def test_experts(rt, H, F, Fs, counts, top):
    E, pairs = len(counts), sum(counts)
    T, g = pairs // top, torch.Generator().manual_seed(H + E)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(pairs, generator=g)][: T * top].view(T, top).int()

    def draw(*shape, std=1.0):
        return (torch.randn(*shape, generator=g) * std).bfloat16().to(rt.device)

    h, gu, down = draw(T, H), draw(E, 2 * F, H, std=H ** -0.5), draw(E, H, F, std=F ** -0.5)
    wts = torch.rand(T, top, generator=g).to(rt.device)
    ids, weights, want = ids.to(rt.device), None, torch.zeros(T, H, dtype=torch.float64, device=rt.device)

    def expert(x, gu, down):
        a, b = (x.double() @ gu.double().T).chunk(2, -1)
        return (a * torch.sigmoid(a) * b) @ down.double().T

    for e in range(E):
        t, k = (ids == e).nonzero(as_tuple=True)
        want.index_add_(0, t, wts[t, k].double()[:, None] * expert(h[t], gu[e], down[e]))
    if Fs:
        weights = (draw(2 * Fs, H, std=H ** -0.5), draw(H, Fs, std=Fs ** -0.5))
        want += expert(h, *weights)
        assert rt.ops.moe_takes_shared(h, top, gu, down, *weights)
    meta = K.make_context(rt, [(0, T)], 16, [[1] * (-(-T // 16))])[0].meta
    assert rt.ops._moe_on_tcgen05(pairs, E, F, h, gu, down)  # (not the tile kernel for few rows)
    out = torch.full((T, H), float("nan"), dtype=rt.dtype, device=rt.device)
    rt.ops.moe_experts(h, ids, wts, gu, down, None, out, meta, **({"shared_weights": weights} if Fs else {}))
    rt.ops.check_status()
    # three roundings to bfloat16 (the activation, a pair's result, the sum): 2^-9 of a value each at most
    assert float((out.double() - want).norm() / want.norm()) < 3 * 2.0 ** -9
    again = torch.empty_like(out)
    rt.ops.moe_experts(h, ids, wts, gu, down, None, again, meta, **({"shared_weights": weights} if Fs else {}))
    assert torch.equal(out, again)


@pytest.mark.parametrize("T", [40, 300])  # 80 and 600 pairs
def test_a_choice_that_names_no_expert_adds_nothing(rt, T):
    """Such a pair stands nowhere in the sorted order: no row is gathered for it and none is added."""
    E, H, F, g = 5, 72, 40, torch.Generator().manual_seed(T)
    ids = torch.randint(0, E, (T, 2), generator=g, dtype=torch.int32)
    ids[::3, 0], ids[1::7, 1], ids[5] = E, -1, 1 << 30
    h, gu, down = (torch.randn(*s, generator=g).bfloat16().to(rt.device) for s in ((T, H), (E, 2 * F, H), (E, H, F)))
    wts = torch.rand(T, 2, generator=g).to(rt.device)
    meta = K.make_context(rt, [(0, T)], 16, [[1] * (-(-T // 16))])[0].meta

    def run(ids, wts):
        out = torch.full((T, H), float("nan"), dtype=rt.dtype, device=rt.device)
        rt.ops.moe_experts(h, ids.to(rt.device), wts, gu, down, None, out, meta)
        rt.ops.check_status()
        return out

    bad = (ids < 0) | (ids >= E)
    assert torch.equal(run(ids, wts), run(ids.masked_fill(bad, 0), wts.masked_fill(bad.to(rt.device), 0.0)))


@pytest.mark.parametrize("T,shared", [(33, False), (127, True)])
def test_results_of_up_to_255_pairs_are_summed_in_float32(rt, T, shared):
    """The second expert takes back all but a 64th of what the first one adds: a result rounded to bfloat16 before the weighted sum would
    put 2^-9 of the whole into the rest."""
    H, F, g = 136, 72, torch.Generator().manual_seed(T)

    def draw(*shape, std=1.0):
        return (torch.randn(*shape, generator=g) * std).bfloat16().to(rt.device)

    h, gu, down = draw(T, H), draw(1, 2 * F, H, std=H ** -0.5).repeat(2, 1, 1), draw(2, H, F, std=F ** -0.5)
    down[1] = (-down[0].float() * (1 + torch.randn(H, F, generator=g).to(rt.device) / 64)).bfloat16()
    weights = (torch.zeros_like(gu[0]), torch.zeros_like(down[0])) if shared else None
    ids = torch.tensor([[0, 1]]).repeat(T, 1).int().to(rt.device)
    out, meta = torch.empty_like(h), K.make_context(rt, [(0, T)], 16, [[1] * (-(-T // 16))])[0].meta
    rt.ops.moe_experts(h, ids, torch.ones(T, 2, device=rt.device), gu, down, None, out, meta, **({"shared_weights": weights} if shared else {}))
    rt.ops.check_status()
    a, b = (h.double() @ gu[0].double().T).chunk(2, -1)
    want = (a * torch.sigmoid(a) * b) @ (down[0].double() + down[1].double()).T
    # the activation and the sum are rounded to bfloat16 (2^-9 each at most); float32 sums of results 64 times as large: 64 * 1e-6
    assert float((out.double() - want).norm() / want.norm()) < 2 * 2.0 ** -9 + 1e-4


@pytest.mark.parametrize("E", [1024, 1025, 12287])
def test_very_many_experts(rt, E):
    """The counts of all experts wait in shared memory beside the stages, of which there are fewer then."""
    T, top, H, F, g = 150, 2, 64, 8, torch.Generator().manual_seed(E)
    ids = torch.randint(0, E, (T, top), generator=g, dtype=torch.int32)
    ids[:70, 0], ids[70:, 1], ids[:70, 1] = 0, E - 1, 1
    h, gu, down = (torch.randn(*s, generator=g).bfloat16().to(rt.device) for s in ((T, H), (E, 2 * F, H), (E, H, F)))
    ids, wts = ids.to(rt.device), torch.rand(T, top, generator=g).to(rt.device)
    assert rt.ops._moe_on_tcgen05(T * top, E, F, h, gu, down)
    out, meta = torch.full_like(h, float("nan")), K.make_context(rt, [(0, T)], 16, [[1] * (-(-T // 16))])[0].meta
    rt.ops.moe_experts(h, ids, wts, gu, down, None, out, meta)
    rt.ops.check_status()
    a, b = torch.einsum("td,tkfd->tkf", h.double(), gu[ids.long()].double()).chunk(2, -1)
    want = torch.einsum("tk,tkf,tkdf->td", wts.double(), a * torch.sigmoid(a) * b, down[ids.long()].double())
    assert float((out.double() - want).norm() / want.norm()) < 3 * 2.0 ** -9


@pytest.mark.parametrize("T", [90, 300])
def test_rows_that_are_no_numbers_and_rows_beyond_the_step(rt, T):
    """Rows that hold an infinity or a NaN beside other experts' and their own expert's rows, in a step whose last ten rows are
    padding (the launch is sized for them, the step's metadata is not): every other row comes out to the bit as without them."""
    E, top, H, F, g = 4, 2, 72, 40, torch.Generator().manual_seed(T)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).int().to(rt.device)
    h, gu, down = (torch.randn(*s, generator=g).bfloat16().to(rt.device) for s in ((T, H), (E, 2 * F, H), (E, H, F)))
    weights, wts = (gu[0] * 0.5, down[0] * 0.5), torch.rand(T, top, generator=g).to(rt.device)
    real = T - 10
    meta = K.make_context(rt, [(0, real)], 16, [[1] * (-(-T // 16))])[0].meta

    def run(h, ids):
        out = torch.full((T, H), 7.0, dtype=rt.dtype, device=rt.device)
        rt.ops.moe_experts(h, ids, wts, gu, down, None, out, meta, shared_weights=weights)
        rt.ops.check_status()
        return out

    want = run(h, ids)
    odd, odd_ids = h.clone(), ids.clone()
    odd[3, 5], odd[17], odd[40, 1], odd[real:] = float("inf"), float("nan"), float("-inf"), float("nan")
    odd_ids[real:] = 1 << 30  # what stands behind the step's rows is never looked at
    got = run(odd, odd_ids)
    rest = [t for t in range(real) if t not in (3, 17, 40)]
    assert torch.equal(got[rest], want[rest]) and bool(torch.isfinite(got[rest]).all())
    assert bool(got[17].isnan().all()) and not bool(torch.isfinite(got[[3, 40]]).all(1).any())
    assert bool((got[real:] == 7.0).all())
