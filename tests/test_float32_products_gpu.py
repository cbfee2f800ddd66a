"""Float32 products of large weights on the tensor cores (three TF32 products, short sums) against float64."""
import pytest
import torch

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
    # A product loses what its two rests were cut by, at most 2^-21 of it, and rest times rest, 2^-22; a run of 32 drops at most an
    # ulp (2^-23) of its sum twelve times; the runs are added with one rounding each.
    bound = (2 ** -21 + 2 ** -22 + 12 * 2 ** -23 + (K / 32 + 4) * 2 ** -24) * (x.double().abs() @ w.double().abs().T)
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
    x[9, 1], w[20, 1] = 3.4028234e38, 1.0 + 2 ** -12  # beyond the largest TF32 number, and a product that overflows
    y, plain = both(rt, x.to(rt.device), w.to(rt.device))
    assert torch.equal(y.isnan(), plain.isnan()) and torch.equal(y.isinf(), plain.isinf())
    odd = ~torch.isfinite(plain)
    assert bool(odd.any()) and torch.equal(y[odd].nan_to_num(), plain[odd].nan_to_num())
