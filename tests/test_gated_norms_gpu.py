"""The gates behind the recurrent layers' scans (norms with a SiLU or sigmoid gate, the convolution's activation): gates that are no
numbers, infinite or far from zero, against the same expression in float64."""
import math

import pytest
import torch

import kernel_utils as K

pytestmark = pytest.mark.gpu
GATES = [math.nan, math.inf, -math.inf, -1e30, -1e4, -104.0, -89.0, -87.5, -87.0, -64.5, -64.0, -1.0, 0.0, 1.0, 64.0, 87.0, 89.0, 1e4]
# float32: a few roundings and sums of up to 1,024 squares; bfloat16, which has 8 significant bits: half a unit of the last one, at
# most 2^-8 of the value, and the float32 part
REL = {"float32": 1e-5, "bfloat16": 2.0 ** -8 + 1e-5}


@pytest.fixture(scope="module")
def rts():
    from atoma_infer_b200.engine.runtime import make_runtime

    return {d: make_runtime(d, "cuda:0") for d in ("float32", "bfloat16")}


def rows(rt, T):
    return K.make_context(rt, [(0, T)], 16, [[1] * (-(-T // 16))])[0]


def sigmoid(g):
    return 1 / (1 + torch.exp(-g.double()))


def silu(g):
    return g.double() * sigmoid(g)


def same(got, want, rel):
    """No numbers and infinities in the same places, everything else within ``rel`` (below 1e-34: gates that count as zero)."""
    got = got.double().cpu()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    ok = want.isfinite()
    assert bool(((got - want)[ok].abs() <= rel * want[ok].abs() + 1e-34).all())


def special_gates(rt, T, n, pad, one_a_row, seed=0):
    """Gates as a slice of wider rows: normal ones, and GATES in turn, in every element or in one of every row."""
    g = torch.Generator().manual_seed(seed)
    wide = torch.randn(T, n + pad, generator=g)
    special = torch.tensor(GATES)
    if one_a_row:
        wide[:, pad + 5] = special[torch.arange(T) % len(GATES)]
    else:
        wide[:, pad:] = special[(torch.arange(T)[:, None] + torch.arange(n)) % len(GATES)]
    return wide.to(rt.dtype)[:, pad:]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("kind", ["sigmoid", "silu"])
@pytest.mark.parametrize("P,pad", [(128, 8), (512, 8), (640, 8), (96, 3)])
def test_gates_behind_a_norm_with_a_weight_per_channel(rts, dtype, kind, P, pad):
    rt, T, heads = rts[dtype], 37, 3
    g = torch.Generator().manual_seed(P)
    o, w = torch.randn(T, heads * P, generator=g), torch.rand(heads * P, generator=g) + 0.5
    gate = special_gates(rt, T, heads * P, pad, False)
    out = torch.empty(T, heads * P, dtype=rt.dtype, device=rt.device)
    rt.ops.head_weight_norm_gate(o.to(rt.device), gate.to(rt.device), w.to(rt.device), 1e-5, out, rows(rt, T).meta, heads, kind=kind)
    v = o.double().view(T, heads, P)
    v = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).reshape(T, -1) * w.double()
    same(out, v * (silu(gate) if kind == "silu" else sigmoid(gate)), REL[dtype])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T", [18, 400])  # (at three heads or parts: below and above the rows from which a warp takes a part)
@pytest.mark.parametrize("which", ["parts", "heads"])
def test_gates_of_the_norms_in_parts_and_per_head(rts, dtype, T, which):
    rt, parts, P = rts[dtype], 3, 128
    g = torch.Generator().manual_seed(T)
    y, w = torch.randn(T, parts * P, generator=g), torch.rand(parts * P, generator=g) + 0.5
    z = special_gates(rt, T, parts * P, 8, which == "parts")
    out = torch.empty(T, parts * P, dtype=rt.dtype, device=rt.device)
    meta, dev = rows(rt, T).meta, lambda t: t.to(rt.device)
    v = y.double().view(T, parts, P)
    if which == "parts":
        rt.ops.gated_group_norm(dev(y), dev(z), dev(w), parts, 1e-5, out, meta)
        v = v * silu(z).view(T, parts, P)
        want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).reshape(T, -1) * w.double()
    else:
        rt.ops.head_norm_gate(dev(y), dev(z), dev(w[:P].contiguous()), 1e-5, out, meta, parts)
        want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w[:P].double()).reshape(T, -1) * silu(z)
    same(out, want, REL[dtype])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_activation_behind_the_convolution(rts, dtype):
    """Two taps of weights 0 and 1: the activation of the rows themselves."""
    rt, T, C = rts[dtype], 21, 64
    ctx = rows(rt, T)
    u = torch.randn(T, C + 8, generator=torch.Generator().manual_seed(1))
    u[-1, 8:] = torch.tensor(GATES)[torch.arange(C) % len(GATES)]  # (the last row: a weight of 0 would pass no numbers on)
    u = u.to(rt.dtype)[:, 8:]
    w = torch.stack([torch.zeros(C), torch.ones(C)])
    out = torch.empty(T, C, dtype=rt.dtype, device=rt.device)
    rt.ops.causal_conv_act(u.to(rt.device), w.to(rt.device), None, torch.zeros(1, 1, C, device=rt.device), ctx, out)
    same(out, silu(u), REL[dtype])


@pytest.mark.parametrize("which", ["parts", "heads", "weights"])
def test_a_float32_row_has_one_order_of_summation(rts, which):
    """Rows alone and among many more (bfloat16 takes other kernels from about a thousand rows on): the same bits."""
    rt, T, parts, P = rts["float32"], 700, 4, 256
    g = torch.Generator().manual_seed(7)
    y, z, w = (torch.randn(*shape, generator=g).to(rt.device) for shape in ((T, parts * P), (T, parts * P + 8), (parts * P,)))

    def run(n):
        out, meta, gate = torch.empty(n, parts * P, device=rt.device), rows(rt, n).meta, z[:n, 8:]
        if which == "parts":
            rt.ops.gated_group_norm(y[:n], gate, w, parts, 1e-5, out, meta)
        elif which == "heads":
            rt.ops.head_norm_gate(y[:n], gate, w[:P].contiguous(), 1e-5, out, meta, parts)
        else:
            rt.ops.head_weight_norm_gate(y[:n], gate, w, 1e-5, out, meta, parts, kind="sigmoid")
        return out

    many = run(T)
    for n in (1, 5, 250):
        assert torch.equal(run(n), many[:n])


@pytest.mark.parametrize("pad", [8, 3])  # gates on and off the boundaries of vector accesses
@pytest.mark.parametrize("length", [4, 124, 128, 132, 256, 260, 512, 516, 1020, 1024, 1028])
@pytest.mark.parametrize("which", ["parts", "heads", "weights"])
def test_norms_of_many_rows(rts, which, length, pad):
    """Rows enough for the kernels in which a warp takes a part or a head, lengths that fill its lanes' loads or leave lanes empty."""
    rt, n = rts["bfloat16"], 3
    T = 8 * torch.cuda.get_device_properties(0).multi_processor_count // n + 17
    g = torch.Generator().manual_seed(length)
    y, w = torch.randn(T, n * length, generator=g), torch.rand(n * length, generator=g) + 0.5
    z = torch.randn(T, n * length + pad, generator=g).to(rt.dtype)[:, pad:]
    out, meta, dev = torch.full((T, n * length), float("nan"), dtype=rt.dtype, device=rt.device), rows(rt, T).meta, lambda t: t.to(rt.device)
    v, gate = y.double().view(T, n, length), silu(z).view(T, n, length)
    if which == "parts":
        rt.ops.gated_group_norm(dev(y), dev(z), dev(w), n, 1e-5, out, meta)
        v = v * gate
        want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w.double().view(n, length)
    else:
        v = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * gate
        if which == "heads":
            rt.ops.head_norm_gate(dev(y), dev(z), dev(w[:length].contiguous()), 1e-5, out, meta, n)
            want = v * w[:length].double()
        else:
            rt.ops.head_weight_norm_gate(dev(y), dev(z), dev(w), 1e-5, out, meta, n, kind="silu")
            want = v * w.double().view(n, length)
    same(out, want.reshape(T, -1), REL["bfloat16"])
