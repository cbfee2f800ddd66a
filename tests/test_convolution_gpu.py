"""The short convolution of prompts, bias and activation, at the edges of its tiles of tokens."""
import pytest
import torch

import kernel_utils as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("taps", [2, 3, 4])
def test_convolution_of_prompts(dtype, taps):
    """Tiles of tokens within one entry, over an entry's end, and at the start of one with and without tokens behind it."""
    from atoma_infer_b200.engine.runtime import make_runtime

    rt = make_runtime(dtype, "cuda:0")
    g, C = torch.Generator().manual_seed(taps), 264
    entries = [(0, 9), (5, 4), (0, 1), (1, 23), (300, 16), (0, 3), (2, 2)]
    ctx, _ = K.make_context(rt, entries, 16, [[1 + i] * 32 for i in range(len(entries))])
    ctx.state_slots.copy_(torch.arange(len(entries), dtype=torch.int32))
    T = sum(n for _, n in entries)
    u, w, b = torch.randn(T, C + 8, generator=g).to(rt.dtype), torch.randn(taps, C, generator=g), torch.randn(C, generator=g)
    ring = torch.randn(len(entries), taps - 1, C, generator=g)
    want, at = torch.zeros(T, C, dtype=torch.float64), 0
    for e, (past, n) in enumerate(entries):
        for t in range(n):
            p = past + t
            acc = b.double()
            for j in range(taps):
                src = p - (taps - 1 - j)
                if src >= 0:
                    acc = acc + w[j].double() * (u[at + src - past, 8:].double() if src >= past else ring[e, src % (taps - 1)].double())
            want[at + t] = acc * torch.sigmoid(acc)
        at += n
    dev = lambda x: x.to(rt.device)  # noqa: E731
    out = torch.full((T, C), float("nan"), dtype=rt.dtype, device=rt.device)
    assert not rt.ops.causal_conv_act(dev(u)[:, 8:], dev(w), dev(b), dev(ring), ctx, out)
    rt.ops.check_status()
    # five float32 roundings and the activation's, or bfloat16's 2^-9 of a result
    assert float(((out.cpu().double() - want).abs() / (want.abs() + 1)).max()) < (2e-6 if dtype == "float32" else 2.0 ** -8)
