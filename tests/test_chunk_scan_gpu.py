"""The scans that run as matrix products over chunks of 128 tokens, at the sizes where that can go wrong: rows of state that fill a
tile partly, columns that leave a part of a block of 64, chunks of 1, 16, 17, 127 and 128 tokens, entries with one chunk beside
entries with several, slots that start on any float.  Against a float64 restatement."""
import ctypes

import pytest
import torch

import kernel_utils as K

pytestmark = pytest.mark.gpu
LENGTHS = [(128,), (129, 1, 16), (127, 17, 256, 300, 2)]
# Sums of a few hundred float32 terms of mixed sign, each good to 2^-24, beside states of the same size: a few 1e-6 of the
# largest value (the bound for the scan in order is 2e-5).
TOL = 1e-5


@pytest.fixture(scope="module")
def rt():
    from atoma_infer_b200.engine.runtime import make_runtime

    return make_runtime("bfloat16", "cuda:0")


def context(rt, lengths):
    ctx, _ = K.make_context(rt, [(3, n) for n in lengths], 16, [[1] * (-(-(n + 3) // 16)) for n in lengths])
    ctx.state_slots.copy_(torch.tensor([len(lengths) - 1 - k for k in range(len(lengths))], dtype=torch.int32))  # not the order of the entries
    return ctx


def scan(q, k, v, log_a, b, S):
    """q, k [T, H, N], v [T, H, P], log_a [T, H] or per row [T, H, N], b [T, H], S [H, N, P], all float64: the outputs and the last
    state."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = torch.exp(log_a[t]).view(q.shape[1], -1, 1) * S + (b[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hnp,hn->hp", S, q[t])
    return out, S


def err(got, want):
    return ((got.double().cpu() - want).abs().max() / want.abs().max()).item()


ENTRY = {"space": ("_mixers", "ssm_chunk_scan"), "memory": ("_matrix_recurrent", "memory_chunk_scan"),
         "decay": ("_recurrent", "gla_row_scan"), "bonus": ("_matrix_recurrent", "bonus_row_scan")}


def both(rt, kind, run, monkeypatch, one_head=0):
    """``run()`` on the chunked kernels and on the one that goes token by token, and that it was so.  ``one_head``: the chunked one
    gets scratch for one head of that many floats."""
    lib, name = getattr(rt.ops, ENTRY[kind][0])(), ENTRY[kind][1]
    entry, calls, got = getattr(lib, name), [], []
    monkeypatch.setattr(lib, name, lambda *args: (calls.append(args), entry(*args))[1])
    for flag in (True, False):
        with monkeypatch.context() as m:
            m.setattr(rt.ops, "matrix_scan", flag)
            if flag and one_head:
                m.setattr(rt.ops, "ROW_SCAN_SCRATCH", one_head + 100)
                m.setattr(lib, name.replace("_row_scan", "_scan_scratch_floats"), lambda *args: 0)
            got.append(run())
        assert len(calls) == 1
    if one_head:
        assert calls[0][-2].value // one_head == 1
    rt.ops.check_status()
    return got


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("heads,P,N,G", [(2, 64, 128, 1), (4, 8, 8, 2), (2, 72, 40, 2), (3, 136, 64, 3), (2, 128, 120, 1)])
def test_state_space_in_matrix_chunks(rt, monkeypatch, lengths, heads, P, N, G):
    g = torch.Generator().manual_seed(heads * P + N + len(lengths))
    T, inner = sum(lengths), heads * P
    xbc = (torch.randn(T, inner + 2 * G * N, generator=g) * 0.7).bfloat16()
    dt = torch.randn(T, heads + 8, generator=g).bfloat16()
    dt_bias, a_log, d = torch.randn(heads, generator=g) - 2, torch.randn(heads, generator=g), torch.randn(heads, generator=g)
    S0 = torch.randn(len(lengths), heads * N * P + 5, generator=g) * 0.5  # an odd slot stride
    want_y, want_s, at = [], {}, 0
    for e, n in enumerate(lengths):
        x = xbc[at:at + n].double()
        step = torch.nn.functional.softplus(dt[at:at + n, :heads].double() + dt_bias.double(), threshold=50)
        xs = x[:, :inner].view(n, heads, P)
        B, C = (x[:, inner + i * G * N:inner + (i + 1) * G * N].view(n, G, N).repeat_interleave(heads // G, 1) for i in (0, 1))
        slot = len(lengths) - 1 - e
        o, S = scan(C, B, xs, -torch.exp(a_log.double()) * step, step, S0[slot, 3:3 + heads * N * P].view(heads, N, P).double())
        want_y.append((o + d.double()[:, None] * xs).reshape(n, inner))
        want_s[slot] = S
        at += n
    want_y, want_s = torch.cat(want_y), torch.stack([want_s[k] for k in range(len(lengths))])
    ctx, dev = context(rt, lengths), lambda t: t.to(rt.device)

    def run():
        state, y = dev(S0.clone()), torch.full((T, inner), float("nan"), device=rt.device)
        mats = state[:, 3:3 + heads * N * P].view(len(lengths), heads, N, P)
        rt.ops.ssm_scan(dev(xbc), dev(dt)[:, :heads], dev(dt_bias), dev(a_log), dev(d), mats, ctx, y, heads=heads, head_dim=P, nstate=N, groups=G)
        assert torch.equal(state[:, :3].cpu(), S0[:, :3]) and torch.equal(state[:, -2:].cpu(), S0[:, -2:])
        return err(y, want_y), err(mats, want_s)

    new, old = both(rt, "space", run, monkeypatch)
    assert max(new) < TOL, (new, old)


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 256), (3, 8, 72), (2, 64, 64), (1, 104, 8)])
def test_matrix_memory_in_matrix_chunks(rt, monkeypatch, lengths, heads, dim, vdim):
    g = torch.Generator().manual_seed(heads * dim + vdim + len(lengths))
    T, cap, nk, nv = sum(lengths), 9.0, heads * dim, heads * vdim
    rows = torch.randn(T, 2 * nk + nv + 8, generator=g).bfloat16()
    logits = torch.randn(T, 2 * heads, generator=g) * 3
    bias = torch.cat([torch.randn(heads, generator=g), 3 + torch.randn(heads, generator=g)])
    up = lambda n: -(-n // 4) * 4  # noqa: E731
    a, b = up(nk * vdim), up(nk)
    S0 = torch.randn(len(lengths), a + b + up(heads) + 4, generator=g) * 0.5
    want, wo, wn, at = {}, [], [], 0
    for e, n in enumerate(lengths):
        x, z = rows[at:at + n].double(), logits[at:at + n].double() + bias.double()
        slot = len(lengths) - 1 - e
        i_g = cap * torch.tanh(z[:, :heads] / cap)
        f_g = -torch.nn.functional.softplus(-cap * torch.tanh(z[:, heads:] / cap))
        m, log_a, w = S0[slot, a + b:a + b + heads].double(), [], []
        for t in range(n):
            new = torch.maximum(f_g[t] + m, i_g[t])
            log_a.append(f_g[t] + m - new)
            w.append(torch.exp(i_g[t] - new))
            m = new
        log_a, w = torch.stack(log_a), torch.stack(w)
        q, k, v = x[:, :nk].view(n, heads, dim) * dim ** -0.5, x[:, nk:2 * nk].view(n, heads, dim), x[:, 2 * nk:2 * nk + nv].view(n, heads, vdim)
        full = torch.cat([v, torch.ones(n, heads, 1, dtype=torch.float64)], -1)  # n is the state of a column of ones
        start = torch.cat([S0[slot, :nk * vdim].view(heads, dim, vdim), S0[slot, a:a + nk].view(heads, dim, 1)], -1).double()
        o, S = scan(q, k, full, log_a, w, start)
        wo.append(o[..., :vdim].reshape(n, nv))
        wn.append(o[..., vdim])
        want[slot] = (S[..., :vdim], S[..., vdim], m)
        at += n
    wo, wn = torch.cat(wo), torch.cat(wn)
    ws = [torch.stack([want[k][j] for k in range(len(lengths))]) for j in range(3)]
    ctx, dev = context(rt, lengths), lambda t: t.to(rt.device)

    def run():
        st = dev(S0.clone())
        state, n_state, m_state = st[:, :nk * vdim].view(-1, heads, dim, vdim), st[:, a:a + nk].view(-1, heads, dim), st[:, a + b:a + b + heads]
        o = torch.full((T, nv), float("nan"), device=rt.device)
        nq, floor = torch.full((T, heads), float("nan"), device=rt.device), torch.full((T, heads), float("nan"), device=rt.device)
        r = dev(rows)
        rt.ops.memory_scan(r[:, :nk], r[:, nk:2 * nk], r[:, 2 * nk:2 * nk + nv], dev(logits), dev(bias), cap, dim ** -0.5, state, n_state, m_state,
                           ctx, o, nq, floor, heads=heads, dim=dim, vdim=vdim)
        return err(o, wo), err(nq, wn), err(state, ws[0]), err(n_state, ws[1]), err(m_state, ws[2])

    new, old = both(rt, "memory", run, monkeypatch)
    assert max(new) < TOL, (new, old)


@pytest.mark.parametrize("lengths", [(128,), (129, 1, 16), (127, 17, 64, 300, 2)])
@pytest.mark.parametrize("heads,dim,vdim", [(3, 128, 256), (2, 8, 72), (2, 64, 64), (1, 104, 8), (2, 40, 16)])
@pytest.mark.parametrize("kind", ["decay", "bonus"])
@pytest.mark.parametrize("rounds", [False, True])
def test_a_decay_per_row_in_matrix_chunks(rt, monkeypatch, lengths, heads, dim, vdim, kind, rounds):
    """Sub-blocks of 16 tokens and triangles of 8 inside chunks of 64; strong decays (rows that forget within a token, whose logs sum
    to thousands within a chunk) beside weak ones; all heads at once, and in rounds of one where scratch is short."""
    g = torch.Generator().manual_seed(heads * dim + vdim + len(lengths))
    T, nk, nv, tau = sum(lengths), heads * dim, heads * vdim, 2.0
    rows = torch.randn(T, 2 * nk + nv + 8, generator=g).bfloat16()
    z, bias, u = torch.randn(T, nk, generator=g) * 2, torch.randn(nk, generator=g), torch.randn(nk, generator=g)
    z[:, 1::7] += 6 if kind == "bonus" else -60  # decays of nearly zero
    z[:, 2::7] -= 9 if kind == "bonus" else -9   # and of nearly one
    S0 = torch.randn(len(lengths), nk * vdim + 5, generator=g) * 0.5
    want, wo, at = {}, [], 0
    for e, n in enumerate(lengths):
        x, x_z = rows[at:at + n].double(), (z[at:at + n].double() + bias.double()).view(n, heads, dim)
        slot = len(lengths) - 1 - e
        q, k, v = x[:, :nk].view(n, heads, dim), x[:, nk:2 * nk].view(n, heads, dim), x[:, 2 * nk:2 * nk + nv].view(n, heads, vdim)
        log_a = -torch.exp(x_z) if kind == "bonus" else -torch.nn.functional.softplus(-x_z, threshold=50) / tau
        S = S0[slot, 3:3 + nk * vdim].view(heads, dim, vdim).double()
        if kind == "decay":
            o, S = scan(q * dim ** -0.5, k, v, log_a, torch.ones(n, heads, dtype=torch.float64), S)
        else:
            o = torch.empty_like(v)
            for t in range(n):
                kv = k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hnp,hn->hp", S + u.double().view(heads, dim, 1) * kv, q[t])
                S = torch.exp(log_a[t])[:, :, None] * S + kv
        wo.append(o.reshape(n, nv))
        want[slot] = S
        at += n
    wo, ws = torch.cat(wo), torch.stack([want[k] for k in range(len(lengths))])
    ctx, dev = context(rt, lengths), lambda t: t.to(rt.device)

    def run():
        st, o, r = dev(S0.clone()), torch.full((T, nv), float("nan"), device=rt.device), dev(rows)
        state = st[:, 3:3 + nk * vdim].view(len(lengths), heads, dim, vdim)
        parts = r[:, :nk], r[:, nk:2 * nk], r[:, 2 * nk:2 * nk + nv]
        if kind == "decay":
            rt.ops.gla_scan(*parts, dev(z), dev(bias), tau, dim ** -0.5, state, ctx, o, heads=heads, dim=dim, vdim=vdim)
        else:
            rt.ops.bonus_scan(*parts, dev(z), dev(bias), dev(u), state, ctx, o, heads=heads, dim=dim, vdim=vdim)
        assert torch.equal(st[:, :3].cpu(), S0[:, :3]) and torch.equal(st[:, -2:].cpu(), S0[:, -2:])
        return err(o, wo), err(state, ws)

    head = 0
    if rounds:
        lib = rt.ops._recurrent() if kind == "decay" else rt.ops._matrix_recurrent()
        x = torch.empty(16, device=rt.device, dtype=torch.bfloat16)
        p, stride = ctypes.c_void_p(x.data_ptr()), ctypes.c_longlong(8)
        head = getattr(lib, ("gla" if kind == "decay" else "bonus") + "_row_scan_head_floats")(p, stride, p, stride, p, stride, p, dim, vdim,
                                                                                               ctx.T // 64 + ctx.S)
    new, old = both(rt, kind, run, monkeypatch, head)
    assert max(new) < TOL, (new, old)


# what is written where before the scan: tensor, token of the step, index in its row (or slot and index), value
ODD = [("v", 150, 3, float("inf")), ("v", 167, 67, float("nan")), ("v", 5, 71, float("-inf")), ("k", 160, 9, float("inf")), ("q", 140, 2, float("-inf")),
       ("state", 0, 77, float("inf")), ("v", 137, 3, float("inf")), ("v", 130, 1, 1e36)]


@pytest.mark.parametrize("odd", ODD, ids=lambda o: f"{o[0]}-{o[1]}-{o[3]}")
@pytest.mark.parametrize("kind,dim", [("space", 64), ("space", 128), ("memory", 128), ("memory", 24), ("decay", 128), ("decay", 64), ("bonus", 40), ("bonus", 128)])
def test_what_is_no_finite_number_reaches_later_tokens_only(rt, monkeypatch, kind, dim, odd):
    """An infinity or no number in a row or a state: the same tokens, columns and states as on the kernel that goes token by token
    (where it stands in the middle of a run of 16, tokens of its run come before and behind it)."""
    what, token, place, value = odd
    heads, vdim, lengths, tau = 2, 72, (129, 1, 16, 200), 2.0
    g = torch.Generator().manual_seed(dim)
    T, nk, nv = sum(lengths), heads * dim, heads * vdim
    ctx, dev = context(rt, lengths), lambda t: t.to(rt.device)
    q, k, v = ((torch.randn(T, n, generator=g) * 0.5).bfloat16() for n in (nk, nk, nv))
    S0 = torch.randn(len(lengths), nk * vdim + 2 * nk + 2 * heads, generator=g) * 0.5
    {"q": q, "k": k, "v": v, "state": S0}[what][token, place] = value
    z, bias, u = torch.randn(T, nk, generator=g), torch.randn(nk, generator=g), torch.randn(nk, generator=g)
    z += -5 if kind == "bonus" else 3  # memories of some tens of tokens: no decay over a chunk is zero
    dt = (torch.randn(T, heads, generator=g) * 0.5 - 4).bfloat16()
    logits = torch.randn(T, 2 * heads, generator=g) + torch.tensor([0.0] * heads + [4.0] * heads)
    zeros, ones = torch.zeros(2 * heads, device=rt.device), torch.ones(heads, device=rt.device)

    def run():
        st, o = dev(S0.clone()), torch.full((T, nv), 7.0, device=rt.device)
        state, more = st[:, :nk * vdim].view(len(lengths), heads, dim, vdim), ()
        if kind == "space":
            rt.ops.ssm_scan(dev(torch.cat([v, k, q], 1)), dev(dt), zeros[:heads], zeros[:heads], ones, state, ctx, o, heads=heads, head_dim=vdim, nstate=dim, groups=heads)
        elif kind == "memory":
            n_state, m_state = st[:, nk * vdim:nk * vdim + nk].view(-1, heads, dim), st[:, nk * vdim + nk:nk * vdim + nk + heads]
            nq, floor = torch.empty(T, heads, device=rt.device), torch.empty(T, heads, device=rt.device)
            rt.ops.memory_scan(dev(q), dev(k), dev(v), dev(logits), zeros, 9.0, dim ** -0.5, state, n_state, m_state, ctx, o, nq, floor,
                               heads=heads, dim=dim, vdim=vdim)
            more = (nq, n_state)
        elif kind == "decay":
            rt.ops.gla_scan(dev(q), dev(k), dev(v), dev(z), dev(bias), tau, dim ** -0.5, state, ctx, o, heads=heads, dim=dim, vdim=vdim)
        else:
            rt.ops.bonus_scan(dev(q), dev(k), dev(v), dev(z), dev(bias), dev(u), state, ctx, o, heads=heads, dim=dim, vdim=vdim)
        return tuple(t.double().cpu() for t in (o, state) + more)

    for new, old in zip(*both(rt, kind, run, monkeypatch)):
        assert torch.equal(new.isnan(), old.isnan())
        assert torch.equal(new.isinf(), old.isinf()) and torch.equal(new[new.isinf()], old[old.isinf()])
        ok = old.isfinite()
        small = ok & (old.abs() < 1e30)  # (beside the largest numbers there are)
        assert bool(((new - old)[small].abs() <= TOL * max(1.0, old[small].abs().max().item())).all())
        assert bool(((new - old)[ok].abs() <= TOL * old[ok].abs().max().item()).all())


@pytest.mark.parametrize("a_log", [30.0, 87.0, 89.0, 120.0])
def test_a_head_that_forgets_everything(rt, monkeypatch, a_log):
    """Rates up to infinity: a state that keeps nothing of the tokens before, beside a head that keeps."""
    heads, P, N, lengths = 2, 64, 64, (200, 16)
    g = torch.Generator().manual_seed(3)
    T = sum(lengths)
    ctx, dev = context(rt, lengths), lambda t: t.to(rt.device)
    xbc = torch.randn(T, heads * (P + 2 * N), generator=g).bfloat16()
    dt = torch.randn(T, heads, generator=g).bfloat16()
    rate, S0 = torch.tensor([a_log, 0.0]), torch.randn(len(lengths), heads, N, P, generator=g)

    def run():
        state, y = dev(S0.clone()), torch.full((T, heads * P), float("nan"), device=rt.device)
        rt.ops.ssm_scan(dev(xbc), dev(dt), dev(torch.zeros(heads)), dev(rate), dev(torch.ones(heads)), state, ctx, y, heads=heads, head_dim=P, nstate=N, groups=heads)
        return y.double().cpu(), state.double().cpu()

    for new, old in zip(*both(rt, "space", run, monkeypatch)):
        assert bool(old.isfinite().all()) and err(new, old) < TOL


def test_more_chunks_than_a_grid_counts(rt):
    """One entry of 130 tokens beside 65,499 single ones: the kernel that goes token by token takes them."""
    P = N = 8
    entries = [(3, 130)] + [(3, 1)] * 65499
    T = sum(n for _, n in entries)
    g = torch.Generator(device=rt.device).manual_seed(5)
    xbc, dt = (torch.randn(T, n, generator=g, device=rt.device).bfloat16() for n in (P + 2 * N, 1))
    S0 = torch.randn(len(entries), 1, N, P, generator=g, device=rt.device)
    one = torch.ones(1, device=rt.device)

    def run(first, rows, count):
        ctx, _ = K.make_context(rt, entries[first:first + count], 16, [[1] * 9] * count)
        state, y = S0[first:first + count].clone(), torch.full((ctx.T, P), float("nan"), device=rt.device)
        rt.ops.ssm_scan(xbc[rows:rows + ctx.T], dt[rows:rows + ctx.T], one - 3, one, one, state, ctx, y, heads=1, head_dim=P, nstate=N, groups=1)
        return y, state

    y, state = run(0, 0, len(entries))
    for first, rows, count in ((0, 0, 1), (1, 130, 200), (len(entries) - 70, T - 70, 70)):
        some_y, some_state = run(first, rows, count)
        n = some_y.shape[0]
        assert err(some_y, y[rows:rows + n].double().cpu()) < TOL and err(some_state, state[first:first + count].double().cpu()) < TOL
