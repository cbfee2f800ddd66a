"""Float32 products of large weights on the tensor cores (three bfloat16 numbers an operand, short sums) against float64."""
import pytest
import torch

import kernel_utils as K_
from atoma_infer_b200.engine.runtime import make_runtime

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    return make_runtime("float32", "cuda:0")


def both(rt, x, w):
    try:
        rt.ops.tc_f32 = True
        y = rt.ops.linear(x, w)
        rt.ops.check_status()
        assert rt.ops._f32_on_tcgen05(x, w, y)  # (else both results are the plain kernel's)
        rt.ops.tc_f32 = False
        return y, rt.ops.linear(x, w)
    finally:
        rt.ops.tc_f32 = True


@pytest.mark.parametrize("M,N,K", [
    (1, 1024, 1024), (16, 1025, 1028), (17, 1151, 1024), (192, 1024, 1052),  # one tile of rows, ragged tiles of w and of k
    (193, 2048, 2048), (385, 1030, 1024),                                    # two and three tiles of rows
    (40, 300, 4100), (333, 2048, 8192),                                      # k cut over two and four blocks, a ragged last part
    (5, 18944, 1024), (700, 2176, 1036),                                     # as many tiles as multiprocessors, more rounds than one
])
def test_products_are_closer_than_one_float32_accumulator(rt, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(rt.device)
    w = (torch.randn(N, K, generator=g) * torch.logspace(-3, 0, N).unsqueeze(1)).to(rt.device)
    y, plain = both(rt, x, w)
    want = x.double() @ w.double().T
    # A product loses lo lo, at most 2^-32 of it; a run of 32 drops at most an ulp (2^-23) of its sum twice, the small terms' sum (2^-7)
    # fourteen times a run; the runs are added with one rounding each, and so are the two sums.
    bound = (2 ** -32 + 2 * 2 ** -23 + 14 * (K / 32 + 1) * 2 ** -30 + (K / 32 + 2) * 2 ** -24) * (x.double().abs() @ w.double().abs().T)
    assert bool(((y.double() - want).abs() <= bound).all())
    assert (y.double() - want).norm() <= (plain.double() - want).norm()
    for m in {0, M // 2, M - 1}:  # a row's bits do not depend on its neighbours
        assert torch.equal(rt.ops.linear(x[m:m + 1].clone(), w)[0], y[m])


@pytest.mark.parametrize("M,N,K", [(20, 1024, 1024), (200, 512, 4096)])
def test_what_is_not_finite_comes_out_as_in_plain_float32(rt, M, N, K):
    g = torch.Generator().manual_seed(7)
    x, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    x[3, 5], x[4, K - 1], x[7, 9] = float("inf"), float("-inf"), float("nan")
    w[11, 5], w[12, 5], w[13, 0] = 0.0, float("inf"), float("nan")
    x[9, 1], w[20, 1] = 3.4028234e38, 1.0 + 2 ** -12  # beyond the scaled range, and a product that overflows
    y, plain = both(rt, x.to(rt.device), w.to(rt.device))
    assert torch.equal(y.isnan(), plain.isnan()) and torch.equal(y.isinf(), plain.isinf())
    odd = ~torch.isfinite(plain)
    assert bool(odd.any()) and torch.equal(y[odd].nan_to_num(), plain[odd].nan_to_num())


@pytest.mark.parametrize("M,N,K", [(70, 1030, 1024), (33, 520, 4100)])
@pytest.mark.parametrize("terms", [0, 1, 2, 3, 8])
def test_rows_of_few_terms_lose_nothing(rt, M, N, K, terms):
    """Rows of x with few numbers that are not zero, where no long sum hides how the operands are held.  0: ones, of which one a row."""
    g = torch.Generator().manual_seed(N + terms)
    w = torch.randn(N, K, generator=g)
    x, at = torch.zeros(M, K), torch.stack([torch.randperm(K, generator=g)[:max(terms, 1)] for _ in range(M)])
    x.scatter_(1, at, torch.randn(M, max(terms, 1), generator=g) if terms else torch.ones(M, 1))
    x, w, at = x.to(rt.device), w.to(rt.device), at.to(rt.device)
    y, plain = both(rt, x, w)
    if not terms:
        assert torch.equal(y, w[:, at[:, 0]].T)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # A term is rounded once, like every sum of two; lo lo (2^-32) is left out and the small terms' sum cut at 2^-23 of their 2^-7.  Terms
    # that share a run of 32 are cut (2^-23), not rounded, where they are added.
    assert bool(((y.double() - want).abs() <= (terms * 2 ** -24 + (terms - 1) * 2 ** -23 * (terms > 1) + 2 ** -28) * size).all())
    assert (y.double() - want).norm() <= 1.1 * (plain.double() - want).norm()


@pytest.mark.parametrize("scale_x,scale_w", [(-126, 40), (-140, 60), (-149, 100), (30, -149), (-100, -20), (-70, -70), (50, 25), (90, -60)])
def test_very_small_and_very_large_numbers(rt, scale_x, scale_w):
    """Subnormal operands and results keep all of their bits; what the scaled sums cannot hold is taken again."""
    M, N, K, g = 40, 1024, 1024, torch.Generator().manual_seed(200 + scale_x)

    def draw(n, scale):  # (whole numbers below 256 at the very bottom of float32's range, else normal ones)
        if scale < -130:
            return (torch.randint(-255, 256, (n, K), generator=g).double() * 2.0 ** scale).float()
        return (torch.randn(n, K, generator=g).double() * 2.0 ** scale).float()

    x, w = draw(M, scale_x).to(rt.device), draw(N, scale_w).to(rt.device)
    y, plain = both(rt, x, w)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = 2 ** -21 * size + 2.0 ** -149  # (the sums as above, and a subnormal result's own rounding)
    assert bool(((y.double() - want).abs() <= bound).all())
    assert (y.double() - want).norm() <= (plain.double() - want).norm() + 2.0 ** -149 * (M * N) ** 0.5


def test_elements_beyond_the_scaled_range_are_the_plain_products(rt):
    g = torch.Generator().manual_seed(9)
    x, w = torch.randn(150, 1024, generator=g), torch.randn(1100, 1024, generator=g)
    x[::2] *= 2.0 ** 85  # sums of about 2^105; below 2^80, where they would not be taken again, is one in 2^25
    w[::3] *= 2.0 ** 15
    x[5, 7] = 2.0 ** 105  # (an operand beyond the range; its products, at most 2^123, are not beyond float32's)
    y, plain = both(rt, x.to(rt.device), w.to(rt.device))
    large = torch.zeros(150, 1100, dtype=torch.bool)
    large[::2, ::3] = large[5] = True
    assert torch.equal(y.cpu()[large], plain.cpu()[large]) and bool(torch.isfinite(y).all())


def test_rows_that_are_no_numbers_cost_no_more_than_the_plain_product(rt):
    """A whole batch of NaN, and one whose NaN stand in rows behind the step's own: those are not taken again."""
    M, N, K, real = 333, 4096, 2048, 300
    x, w = torch.full((M, K), float("nan"), device=rt.device), torch.randn(N, K, device=rt.device)
    meta = K_.make_context(rt, [(0, real)], 16, [[1] * 20])[0].meta
    fine = torch.randn(M, K, device=rt.device)
    padded = fine.clone()
    padded[real:] = float("nan")

    def time(x, tc, meta=None):
        rt.ops.tc_f32, best = tc, 1e9
        try:
            for _ in range(5):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                y = rt.ops.linear(x, w, meta=meta)
                b.record()
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(b))
        finally:
            rt.ops.tc_f32 = True
        return best, y

    plain = time(x, False)[0]
    t, y = time(x, True)
    assert bool(y.isnan().all()) and t < 3 * plain  # (a lane an element: over 50 times)
    t, y = time(padded, True, meta)
    assert torch.equal(y[:real], time(fine, True)[1][:real]) and t < plain
