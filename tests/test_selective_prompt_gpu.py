"""The selective scan of prompts in one pass (kernels/selective_prompt.cuh) against the plain implementation in float64."""
import pytest
import torch

import plain_bumolix as PB
from test_bumolix_kernels_gpu import _context

from atoma_infer_b200.csrc import ops as O
from atoma_infer_b200.engine.runtime import make_runtime

pytestmark = pytest.mark.gpu


def takes(rt, u, dt, bc, z, out, C, N):
    """Whether these inputs reach the kernel (else the call would fall back to the others)."""
    (up, us), (bp, bs), (zp, zs) = (rt.ops._rows(t, "takes") for t in (u, bc, z))
    return rt.ops._recurrent().selective_scan_prompt_takes(up, us, O._p(dt), bp, bs, zp, zs, O._code(u), O._p(out), C, N)


# entries without a token, one token, a tile's edges and one beyond, several tiles; channels that fill no block, one, and more
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("C,N,lens", [(8, 16, [1]), (40, 8, [31, 0, 32, 33]), (32, 16, [64, 3, 65]), (72, 16, [257, 1, 96]), (1032, 8, [40])])
def test_one_pass_equals_the_plain_scan(dtype, C, N, lens):
    rt = make_runtime(dtype, "cuda:0")
    g = torch.Generator().manual_seed(C + N + len(lens))
    T, n = sum(lens), len(lens)
    row = torch.randn(T, 2 * C + 8 + 2 * N, generator=g).to(rt.dtype)
    dt, dt_bias = 2 * torch.randn(T, C, generator=g), torch.randn(C, generator=g) - 1.0
    a_log, d_skip = 1.5 * torch.randn(C, N, generator=g), torch.randn(C, generator=g)
    wide = torch.randn(n + 2, 6 + C * N + 2, generator=g)  # a state inside wider slots, not all of them used
    slots = [n + 1 - i for i in range(n)]
    dev = wide.to(rt.device)
    out = torch.full((T, C), float("nan"), dtype=rt.dtype, device=rt.device)
    x, ctx = row.to(rt.device), _context(rt, [(i, 0, m) for i, m in enumerate(lens)], slots)
    rt.ops.selective_prompt = True
    u, z, bc = x[:, :C], x[:, C:2 * C], x[:, 2 * C + 8:]
    assert takes(rt, u, dt.to(rt.device), bc, z, out, C, N)
    rt.ops.selective_scan(u, dt.to(rt.device), dt_bias.to(rt.device), bc, z, a_log.to(rt.device), d_skip.to(rt.device),
                          dev[:, 6:6 + C * N].unflatten(1, (C, N)), ctx, out, inner=C, nstate=N)
    rt.ops.check_status()
    at, r = 0, row.double()
    for i, m in enumerate(lens):
        S = wide[slots[i], 6:6 + C * N].double().view(C, N)
        A, rows = -torch.exp(a_log.double()), slice(at, at + m)
        for t in range(at, at + m):
            step = PB.softplus(dt[t].double() + dt_bias.double())
            S = torch.exp(step[:, None] * A) * S + (step * r[t, :C])[:, None] * r[t, 2 * C + 8:2 * C + 8 + N]
            y = ((S * r[t, 2 * C + 8 + N:]).sum(1) + d_skip.double() * r[t, :C]) * PB.silu(r[t, C:2 * C])
            # float32 throughout, a few roundings a token of a memory of some tens of tokens: 1e-5; bfloat16: the result's own rounding
            tol = 1e-5 if dtype == "float32" else 2 ** -8
            assert ((out[t].double().cpu() - y).abs() <= tol * (y.abs() + 1)).all(), (i, t - at)
        kept = dev[slots[i], 6:6 + C * N].double().cpu().view(C, N)
        assert ((kept - S).abs() <= 1e-5 * (S.abs() + 1)).all()
        at += m
    untouched = [s for s in range(n + 2) if s not in slots]
    assert torch.equal(dev[untouched].cpu(), wide[untouched]) and torch.equal(dev[:, :6].cpu(), wide[:, :6]) and torch.equal(dev[:, -2:].cpu(), wide[:, -2:])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("N,one_sign", [(16, False), (16, True), (8, False), (8, True)])  # one_sign: an infinite state gives infinite results
def test_what_is_not_finite_reaches_what_it_reaches_in_order(dtype, N, one_sign):
    """Against the kernel that takes the tokens in order, too: the one in chunks multiplies an infinite state by the whole decay of
    a chunk, and where that is 0 it makes a NaN of what token by token stays infinite."""
    rt = make_runtime(dtype, "cuda:0")
    g = torch.Generator().manual_seed(5)
    C, T = 64, 150
    row, dt = torch.randn(T, 2 * C + 2 * N, generator=g), torch.randn(T, C, generator=g)
    if one_sign:
        row[:, 2 * C:].abs_()
    row[40, 3], row[60, C + 5], row[90, 2 * C + 4], dt[20, 7], dt[30, 9] = float("inf"), float("nan"), float("inf"), float("inf"), float("-inf")
    a_log = torch.randn(C, N, generator=g)
    a_log[11, 2], a_log[12] = float("inf"), float("-inf")
    x = row.to(rt.dtype).to(rt.device)
    rt.ops.SCAN_CHUNK_FROM = 1 << 30
    results = []
    u, z, bc = x[:, :C], x[:, C:2 * C], x[:, 2 * C:]
    assert takes(rt, u, dt.to(rt.device), bc, z, torch.empty((T, C), dtype=rt.dtype, device=rt.device), C, N)
    for one_pass in (True, False):
        rt.ops.selective_prompt = one_pass
        state = torch.zeros((1, C, N), device=rt.device)
        out = torch.empty((T, C), dtype=rt.dtype, device=rt.device)
        rt.ops.selective_scan(x[:, :C], dt.to(rt.device), torch.zeros(C, device=rt.device), x[:, 2 * C:], x[:, C:2 * C], a_log.to(rt.device),
                              torch.ones(C, device=rt.device), state, _context(rt, [(0, 0, T)], [0]), out, inner=C, nstate=N)
        results.append((out.float().cpu(), state.cpu()))
    assert not one_sign or bool(results[1][0][50, 3].isinf())
    for new, old in zip(*results):
        assert torch.equal(new.isnan(), old.isnan())
        assert torch.equal(new.isinf(), old.isinf()) and torch.equal(new[new.isinf()], old[old.isinf()])


def test_float32_bits_do_not_depend_on_the_other_requests():
    """A request's 40 tokens alone and beside so many others that another kernel would be the shorter way."""
    rt = make_runtime("float32", "cuda:0")
    g = torch.Generator().manual_seed(3)
    C, N, n = 4096, 16, 40
    a_log, d_skip, dt_bias = (torch.randn(*s, generator=g).to(rt.device) for s in ((C, N), (C,), (C,)))
    lens = [n] + [1, 30, 64, 2] * 10
    T = sum(lens)
    row, dt = torch.randn(T, 2 * C + 2 * N, generator=g).to(rt.device), torch.randn(T, C, generator=g).to(rt.device)

    def run(lens):
        t = sum(lens)
        state, out = torch.zeros((len(lens), C, N), device=rt.device), torch.empty((t, C), device=rt.device)
        ctx = _context(rt, [(i, 0, m) for i, m in enumerate(lens)], list(range(len(lens))))
        rt.ops.selective_scan(row[:t, :C], dt[:t], dt_bias, row[:t, 2 * C:], row[:t, C:2 * C], a_log, d_skip, state, ctx, out, inner=C, nstate=N)
        return out[:n], state[0]

    for alone, beside in zip(run([n]), run(lens)):
        assert torch.equal(alone, beside)
