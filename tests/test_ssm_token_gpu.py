"""The state-space mixer's decode step in two launches, beside the convolution, the scan in order and the gated norm as kernels of their
own: every column count, the most rows and odd numbers of them, one to four taps, first tokens, slots out of order."""
import pytest
import torch

import kernel_utils as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,P,N,G,taps", [(16, 64, 128, 2, 4), (8, 64, 72, 1, 3), (6, 32, 250, 2, 4), (3, 32, 40, 3, 2), (4, 128, 64, 2, 4),
                                              (2, 128, 33, 2, 1), (5, 64, 8, 1, 4), (14, 64, 127, 2, 4)])
def test_against_three_kernels(dtype, heads, P, N, G, taps):
    from atoma_infer_b200.engine.runtime import make_runtime

    rt = make_runtime(dtype, "cuda:0")
    ops, dev = rt.ops, rt.device
    g = torch.Generator().manual_seed(heads * N)
    past = [0, 1, 2, 57, 400]
    S, inner, ch = len(past), heads * P, heads * P + 2 * G * N
    rows = -(-(ch + inner + heads) // 8) * 8  # (wide rows; some slices start on odd elements)
    ctx, _ = K.make_context(rt, [(c, 1) for c in past], 16, [[1 + i] * 32 for i in range(S)])
    assert ctx.decode_only and ctx.T == ctx.S
    ctx.state_slots.copy_(torch.tensor([3, 0, 4, 1, 2], dtype=torch.int32))

    def f(*shape, std=1.0, mean=0.0):
        return (torch.randn(*shape, generator=g) * std + mean).to(dev)

    proj = f(S, rows).to(rt.dtype)
    z, u, dt = proj[:, :inner], proj[:, inner:inner + ch], proj[:, inner + ch:inner + ch + heads]
    conv_w, conv_b, dt_bias, a_log, d, w = f(taps, ch, std=0.3), f(ch, std=0.1), f(heads, mean=-3), f(heads, std=0.5), f(heads), f(inner, std=0.1, mean=1)
    ring_floats = -(-(taps - 1) * ch // 4) * 4
    state = f(S, ring_floats + heads * N * P, std=0.5)

    def parts(s):
        ring = s[:, :(taps - 1) * ch].view(S, taps - 1, ch) if taps > 1 else None
        return ring, s[:, ring_floats:].view(S, heads, N, P)

    ours, theirs = state.clone(), state.clone()
    got, want = (torch.full((S, inner), float("nan"), dtype=rt.dtype, device=dev) for _ in range(2))
    assert ops.ssm_token_step(u, z, dt, conv_w, conv_b, parts(ours)[0], dt_bias, a_log, d, parts(ours)[1], w, G, G, 1e-5, ctx, got)
    xbc, y = torch.empty(S, ch, dtype=rt.dtype, device=dev), torch.empty(S, inner, device=dev)
    if not ops.causal_conv_act(u, conv_w, conv_b, parts(theirs)[0], ctx, xbc):
        ops.causal_conv_save(u, parts(theirs)[0], ctx, taps)
    ops.ssm_scan(xbc, dt, dt_bias, a_log, d, parts(theirs)[1], ctx, y, heads=heads, head_dim=P, nstate=N, groups=G)
    ops.gated_group_norm(y, z, w, G, 1e-5, want, ctx.meta)
    ops.check_status()
    # the same products and roundings; sums over N rows in another order: sqrt(N) 2^-24 of the terms and, in bfloat16, now and then the
    # neighbouring number (2^-8 of a value, of which the 2-norm sees few)
    assert torch.equal(ours[:, :ring_floats], theirs[:, :ring_floats])
    assert float((ours - theirs).norm() / theirs.norm()) < 1e-6
    assert float((got.double() - want.double()).norm() / want.double().norm()) < (2e-6 if dtype == "float32" else 1e-3)


def test_other_steps_are_left_alone():
    from atoma_infer_b200.engine.runtime import make_runtime

    rt = make_runtime("bfloat16", "cuda:0")
    t = torch.zeros(4, 512, dtype=rt.dtype, device=rt.device)
    state = torch.zeros(4, 2, 16, 64, device=rt.device)
    one = torch.zeros(512, device=rt.device)

    def takes(entries, norm_groups=1):
        ctx, _ = K.make_context(rt, entries, 16, [[1 + i] for i in range(len(entries))])
        return rt.ops.ssm_token_step(t[:ctx.T, :160], t[:ctx.T, :128], t[:ctx.T, :2], one[:160].view(1, 160), None, None, one[:2], one[:2], one[:2], state,
                                     one[:128], 1, norm_groups, 1e-5, ctx, torch.zeros_like(t[:ctx.T, :128]))

    assert takes([(3, 1), (4, 1)])
    assert not takes([(0, 2), (4, 1)]) and not takes([(3, 1)], norm_groups=3)


class Step:
    """Five requests' tokens, in slots out of order, with rows of their own and a state that both ways start from."""

    def __init__(self, rt, heads, P, N, G, taps, seed):
        g, dev = torch.Generator().manual_seed(seed), rt.device
        self.rt, self.sizes, self.past = rt, (heads, P, N, G, taps), [0, 1, 2, 57, 400]
        S, inner, ch = len(self.past), heads * P, heads * P + 2 * G * N
        self.ctx, _ = K.make_context(rt, [(c, 1) for c in self.past], 16, [[1 + i] * 32 for i in range(S)])
        self.slots = [3, 0, 4, 1, 2]
        self.ctx.state_slots.copy_(torch.tensor(self.slots, dtype=torch.int32))

        def f(*shape, std=1.0, mean=0.0):
            return (torch.randn(*shape, generator=g) * std + mean).to(dev)

        self.proj = f(S, -(-(2 * inner + 2 * G * N + heads) // 8) * 8).to(rt.dtype)
        self.z, self.u, self.dt = self.proj[:, :inner], self.proj[:, inner:inner + ch], self.proj[:, inner + ch:inner + ch + heads]
        self.conv_w, self.conv_b, self.dt_bias = f(taps, ch, std=0.3), f(ch, std=0.1), f(heads, mean=-3)
        self.a_log, self.d, self.w = f(heads, std=0.5), f(heads), f(inner, std=0.1, mean=1)
        self.ring, self.state = f(S, taps - 1, ch), f(S, heads, N, P, std=0.5)

    def two_launches(self):
        heads, P, N, G, taps = self.sizes
        ring, state, out = self.ring.clone(), self.state.clone(), torch.empty(len(self.past), heads * P, dtype=self.rt.dtype, device=self.rt.device)
        assert self.rt.ops.ssm_token_step(self.u, self.z, self.dt, self.conv_w, self.conv_b, ring, self.dt_bias, self.a_log, self.d, state, self.w, G, G,
                                          1e-5, self.ctx, out)
        self.rt.ops.check_status()
        return out, state, ring

    def three_kernels(self):
        heads, P, N, G, taps = self.sizes
        ops, ring, state = self.rt.ops, self.ring.clone(), self.state.clone()
        xbc, y = torch.empty_like(self.u, memory_format=torch.contiguous_format), torch.empty(len(self.past), heads * P, device=self.rt.device)
        out = torch.empty(len(self.past), heads * P, dtype=self.rt.dtype, device=self.rt.device)
        if not ops.causal_conv_act(self.u, self.conv_w, self.conv_b, ring, self.ctx, xbc):
            ops.causal_conv_save(self.u, ring, self.ctx, taps)
        ops.ssm_scan(xbc, self.dt, self.dt_bias, self.a_log, self.d, state, self.ctx, y, heads=heads, head_dim=P, nstate=N, groups=G)
        ops.gated_group_norm(y, self.z, self.w, G, 1e-5, out, self.ctx.meta)
        return out, state, ring

    def exact(self):
        """The same in 64 bits, without a rounding on the way."""
        heads, P, N, G, taps = self.sizes
        outs, state, ring, R = [], self.state.double(), self.ring.double(), taps - 1
        for e, p in enumerate(self.past):
            s, u = self.slots[e], self.u[e].double()
            acc = self.conv_b.double() + self.conv_w[R].double() * u
            for back in range(1, R + 1):
                if p - back >= 0:
                    acc = acc + self.conv_w[R - back].double() * ring[s, (p - back) % R]
            ring[s, p % R] = u
            x, B, C = (acc * torch.sigmoid(acc)).split([heads * P, G * N, G * N])
            x, B, C = x.view(heads, P), *(t.view(G, N).repeat_interleave(heads // G, 0) for t in (B, C))
            step = torch.nn.functional.softplus(self.dt[e].double() + self.dt_bias.double())
            decay = torch.exp(-torch.exp(self.a_log.double()) * step)
            state[s] = decay[:, None, None] * state[s] + torch.einsum("hn,hp->hnp", B, step[:, None] * x)
            y = (torch.einsum("hnp,hn->hp", state[s], C) + self.d.double()[:, None] * x).reshape(-1)
            z = self.z[e].double()
            v = (y * z * torch.sigmoid(z)).view(G, -1)
            outs.append((v / (v.square().mean(1, keepdim=True) + 1e-5).sqrt()).reshape(-1) * self.w.double())
        return torch.stack(outs), state, ring


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,P,N,G,taps", [(16, 64, 128, 2, 4), (6, 32, 250, 2, 4), (4, 128, 64, 2, 2), (14, 64, 37, 7, 3)])
def test_against_64_bits(dtype, heads, P, N, G, taps):
    from atoma_infer_b200.engine.runtime import make_runtime

    step = Step(make_runtime(dtype, "cuda:0"), heads, P, N, G, taps, seed=heads + N)
    got, want = step.two_launches(), step.exact()
    assert torch.equal(got[2].double(), want[2])
    # float32: sums of up to 250 terms, 250^0.5 2^-24 and exponentials of a few 2^-24; bfloat16: x, B and C are rounded behind the
    # convolution and the result once more, 2^-9 of a value each at most
    for a, b in zip(got[:2], want[:2]):
        assert float((a.double() - b).norm() / b.norm()) < (2e-6 if dtype == "float32" else 4 * 2.0 ** -9)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_what_is_not_finite(dtype):
    """Infinities and NaN in a row, a step size and a state: where the three kernels have them, and nowhere else."""
    from atoma_infer_b200.engine.runtime import make_runtime

    heads, P, N, G = 4, 64, 128, 2
    step = Step(make_runtime(dtype, "cuda:0"), heads, P, N, G, 4, seed=1)
    inner = heads * P
    step.u[0, 5], step.u[1, inner + 3], step.dt[2, 1] = float("inf"), float("nan"), float("inf")  # x of a head, B of a group, a step size
    step.state[step.slots[3], 2, 7, 9], step.state[step.slots[4], 0, 0, 0], step.ring[step.slots[4], 1, 70] = float("-inf"), float("nan"), float("inf")
    for a, b in zip(step.two_launches(), step.three_kernels()):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf()) and not bool(torch.isfinite(a).all())
        assert bool(torch.isfinite(a).any())
        if dtype == "float32":
            assert torch.equal(a.nan_to_num(), b.nan_to_num())


@pytest.mark.parametrize("heads,P,N,G", [(64, 64, 128, 8), (64, 32, 100, 4), (48, 128, 64, 3), (64, 64, 20, 1)])
def test_float32_bits_do_not_depend_on_the_other_requests(heads, P, N, G):
    """A request's token alone, among others at the two sides of where the step stops being taken, and beside a prompt: the layer's
    output and state are the same to the bit."""
    from atoma_infer_b200.engine.runtime import make_runtime
    from atoma_infer_b200.parts.ssm import Mamba2Mixer
    from atoma_infer_b200.cache.spec import LayerCache

    rt = make_runtime("float32", "cuda:0")
    g, dev, H, taps = torch.Generator().manual_seed(P + N), rt.device, 192, 4
    inner, ch = heads * P, heads * P + 2 * G * N

    def f(*shape, std=1.0, mean=0.0):
        return (torch.randn(*shape, generator=g) * std + mean).to(dev)

    part = Mamba2Mixer({"hidden": H, "heads": heads, "head_dim": P, "state": N, "groups": G, "taps": taps, "norm_groups": G, "eps": 1e-5}, "p")
    part.bind({"p.in": f(inner + ch + heads, H, std=H ** -0.5), "p.conv": f(ch, taps, std=0.3), "p.conv.b": f(ch, std=0.1),
               "p.dt_bias": f(heads, mean=-3), "p.A_log": f(heads, std=0.5), "p.D": f(heads), "p.norm": f(inner, std=0.1, mean=1),
               "p.o": f(H, inner, std=inner ** -0.5)}, rt)
    most = 14 * rt.ops.num_sms // heads  # (more than any limit of the rule)
    x, kept = f(most + 3, H), f(most + 3, part.state_bytes() // 4, std=0.5)

    def run(lens):
        """Requests of one token each (row i of x for request i), the last one of lens[-1] tokens."""
        ctx, _ = K.make_context(rt, [(50 + i, n) for i, n in enumerate(lens)], 16, [[1 + i] * 32 for i in range(len(lens))])
        state = kept[:len(lens)].clone()
        rows = torch.cat([x[:len(lens) - 1], x[len(lens) - 1:len(lens)].repeat(lens[-1], 1)])
        cache = LayerCache(group=-1, pages=None, num_pages=0, page_size=16, writes=False, state=state.view(torch.uint8))
        y = part.forward(rows, ctx, cache)
        rt.ops.check_status()
        return y, state

    want_y, want_state = run([1])
    for lens in ([1] * 2, [1] * 9, [1] * most, [1] * (most + 1), [1] * (most + 3), [1, 1, 40]):
        y, state = run(lens)
        assert torch.equal(y[0], want_y[0]) and torch.equal(state[0], want_state[0]), len(lens)
