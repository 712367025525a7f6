"""The recurrences that work 32 tokens at a time, where their chain takes two runs of 16 columns a block (more blocks of one run than SMs), against the
recurrences in float64; the rule with a decay per channel with short portions that go token by token beside long ones, and with tokens that
are not finite."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def step(lengths):
    offsets, positions, item_of = [0], [], []
    for i, n in enumerate(lengths):
        offsets.append(offsets[-1] + n)
        positions += range(7 * i, 7 * i + n)
        item_of += [i] * n
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    return types.SimpleNamespace(positions=dev(positions), token_item=dev(item_of), item_start=dev(offsets), slots=dev(list(range(len(lengths)))[::-1]),
                                 num_items=len(lengths), max_new_tokens=max(lengths), items=[types.SimpleNamespace(start=0, end=n) for n in lengths]), offsets


class Channel:
    """Inputs of the rule with a decay per channel (no convolution behind the projection: one tap), and the rule itself."""

    def __init__(self, lengths, groups, heads, dim, vdim, dtype, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
        self.sizes, self.lengths = dict(groups=groups, heads=heads, dim=dim, vdim=vdim), lengths
        self.ctx, self.offsets = step(lengths)
        t, self.c = sum(lengths), 2 * groups * dim + heads * vdim
        self.proj, self.taps = rnd(t, self.c + heads).to(dtype), 0.5 + rnd(self.c, 1).abs()
        self.decay = torch.rand(t, heads, dim, generator=g, device="cuda") ** 0.1
        self.decay[::5, :, ::3], self.decay[1::7, :, 1::4] = 0.0, 1.0
        self.held = 0.3 * rnd(len(lengths), heads * dim * vdim)

    def run(self, proj=None, decay=None):
        from prefixserve_b200 import ops
        state = self.held.clone()
        proj, decay = self.proj if proj is None else proj, self.decay if decay is None else decay
        return ops.channel_delta_rule(proj, self.c, decay.view(len(proj), -1), self.taps, state, self.ctx, **self.sizes).double(), state

    def exact(self):
        z = self.sizes
        groups, heads, dim, vdim = z["groups"], z["heads"], z["dim"], z["vdim"]
        u = torch.nn.functional.silu(self.proj[:, : self.c].double() * self.taps[:, 0].double())
        unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        q, k = (unit(u[:, a: a + groups * dim].view(-1, groups, dim)).repeat_interleave(heads // groups, 1) for a in (0, groups * dim))
        v, beta, out, state = u[:, 2 * groups * dim:].view(-1, heads, vdim), torch.sigmoid(self.proj[:, self.c:].double()), [], []
        for i, n in enumerate(self.lengths):
            m = self.held[len(self.lengths) - 1 - i].double().view(heads, dim, vdim)
            for t in range(self.offsets[i], self.offsets[i] + n):
                m = m * self.decay[t].double()[:, :, None]
                m = m + k[t, :, :, None] * (beta[t, :, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], m)))[:, None]
                out.append(torch.einsum("hd,hdv->hv", q[t] * dim ** -0.5, m))
            state.append(m.reshape(-1))
        return torch.stack(out), torch.stack(state[::-1])


# 160 blocks of 16 columns and more on 148 SMs, 80 of 32; the last columns' block not full
@pytest.mark.parametrize("heads, dim, vdim, lengths, dtype", [(20, 128, 64, [70, 33], torch.bfloat16), (12, 33, 52, [31, 32, 40, 100], torch.float32),
                                                              (30, 64, 41, [64, 26], torch.bfloat16)])
def test_two_runs_of_columns_decay_per_channel(heads, dim, vdim, lengths, dtype):
    case = Channel(lengths, 2, heads, dim, vdim, dtype, dim)
    out, state = case.run()
    want, held = case.exact()
    assert (out - want).abs().max() < 2e-5 * want.abs().max() and (state.double() - held).abs().max() < 2e-5 * held.abs().max()


@pytest.mark.parametrize("heads, dim, vdim, lengths", [(20, 128, 64, [70, 8]), (40, 32, 20, [9, 97, 33])])
def test_two_runs_of_columns_decay_per_head(heads, dim, vdim, lengths):
    from prefixserve_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(dim)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx, offsets = step(lengths)
    t, c = sum(lengths), 2 * 2 * dim + heads * vdim
    proj, ba, taps = rnd(t, c + heads * vdim).bfloat16(), rnd(t, 2 * heads), 0.5 + rnd(c, 1).abs()
    a_log, dt_bias, held = rnd(heads) - 1, rnd(heads) - 1, 0.3 * rnd(len(lengths), heads * dim * vdim)
    state = held.clone()
    out = ops.delta_rule(proj, ba, taps, a_log, dt_bias, torch.ones(vdim, device="cuda"), state, ctx, groups=2, heads=heads, dim=dim, vdim=vdim, eps=1e-5)
    u = torch.nn.functional.silu(proj[:, :c].double() * taps[:, 0].double())
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(u[:, a: a + 2 * dim].view(-1, 2, dim)).repeat_interleave(heads // 2, 1) for a in (0, 2 * dim))
    v, beta = u[:, 4 * dim:].view(-1, heads, vdim), torch.sigmoid(ba[:, :heads].double())
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(ba[:, heads:].double() + dt_bias.double()))
    for i, n in enumerate(lengths):
        m = held[len(lengths) - 1 - i].double().view(heads, dim, vdim)
        for j in range(offsets[i], offsets[i] + n):
            m = m * decay[j, :, None, None]
            m = m + k[j, :, :, None] * (beta[j, :, None] * (v[j] - torch.einsum("hd,hdv->hv", k[j], m)))[:, None]
            o = torch.einsum("hd,hdv->hv", q[j] * dim ** -0.5, m)
            want = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * torch.nn.functional.silu(proj[j, c:].double()).view(heads, vdim)
            # float32 sums of numbers around one, divided by a root mean square that may be small; the result in bfloat16
            assert ((out[j].double().view(heads, vdim) - want).abs() <= 1e-4 + 2.0 ** -8 * want.abs()).all(), j
        assert (state[len(lengths) - 1 - i].double().view_as(m) - m).abs().max() < 2e-5 * m.abs().max()


@pytest.mark.parametrize("heads, dim, vdim, lengths", [(20, 128, 64, [96, 33]), (24, 36, 44, [100, 32, 63])])
def test_two_runs_of_columns_linear_attention(heads, dim, vdim, lengths):
    from prefixserve_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(dim)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx, offsets = step(lengths)
    t = sum(lengths)
    proj, alpha, held = rnd(t, heads * (2 * dim + vdim)).bfloat16(), torch.sigmoid(rnd(t, heads * dim)) ** 0.25, rnd(len(lengths), heads * dim * vdim)
    state = held.clone()
    out = ops.linear_attention(proj, alpha, state, ctx, heads=heads, dim=dim, vdim=vdim).double()
    p, a = proj.double(), alpha.double().view(t, heads, dim, 1)
    q, k, v = p[:, : heads * dim].view(t, heads, dim), p[:, heads * dim: 2 * heads * dim].view(t, heads, dim), p[:, 2 * heads * dim:].view(t, heads, vdim)
    for i, n in enumerate(lengths):
        m = held[len(lengths) - 1 - i].double().view(heads, dim, vdim)
        for j in range(offsets[i], offsets[i] + n):
            m = a[j] * m + k[j, :, :, None] * v[j, :, None]
            want = torch.einsum("hd,hdv->hv", q[j], m) * dim ** -0.5
            assert (out[j] - want).abs().max() <= 2e-5 * max(1.0, float(want.abs().max())), j
        assert (state[len(lengths) - 1 - i].double().view_as(m) - m).abs().max() < 2e-5 * m.abs().max()


@pytest.mark.parametrize("short, apart", [([1] * 70, True), ([7, 3], False), ([1], False)])
def test_short_portions_beside_long_ones(short, apart):
    """Many short portions go token by token, a few in chunks like the long ones."""
    from prefixserve_b200.ops import library
    case = Channel([50, *short, 24], 2, 4, 64, 96, torch.bfloat16, len(short))
    before = library.launch_counts.copy()
    out, state = case.run()
    taken = library.launch_counts - before
    assert taken["channel_delta_chunks"] == 1 and taken["channel_delta_rule"] == apart
    want, held = case.exact()
    assert (out - want).abs().max() < 2e-5 * want.abs().max() and (state.double() - held).abs().max() < 2e-5 * held.abs().max()


@pytest.mark.parametrize("what", ["value", "key", "query", "decay"])
def test_a_token_that_is_not_finite_reaches_later_tokens_only(what):
    groups, heads, dim, vdim, bad = 2, 4, 128, 64, 45
    case = Channel([100, 40], groups, heads, dim, vdim, torch.bfloat16, 3)
    clean, _ = case.run()
    proj, decay, nan = case.proj.clone(), case.decay.clone(), float("nan")
    if what == "value":
        proj[bad, 2 * groups * dim + 3] = float("inf")                 # a number of the first head
    elif what == "decay":
        decay[bad, 0, 5] = nan
    else:
        proj[bad, 5 + (groups * dim if what == "key" else 0)] = nan    # the first group: heads 0 and 1
    out, state = case.run(proj, decay)
    state, hit = state.view(2, heads, dim, vdim), 2 if what in ("key", "query") else 1
    near = lambda a, b: ((a - b).abs() <= 2e-5 * (1 + b.abs())).all()   # sums made again in another order
    assert torch.isfinite(out[:bad]).all() and near(out[:bad], clean[:bad]) and near(out[100:], clean[100:]) and near(out[:, hit:], clean[:, hit:])
    assert not torch.isfinite(out[bad, :hit]).all(-1).any() and torch.isfinite(state[0]).all() and torch.isfinite(state[1, hit:]).all()
    if what != "query":
        assert not torch.isfinite(out[99, :hit]).all(-1).any() and not torch.isfinite(state[1, :hit].flatten(1)).all(1).any()


# Two runs of columns a block (as above), and one.  Read-outs and states lie 0.6e-7 to 2.1e-7 from float64 (norm of the difference over norm), with what is in front
# of the rule; numbers in two terms instead of three would be off by some 2^-18 = 4e-6.
CLOSE = 4e-7


def off(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("heads, vdim", [(20, 64), (4, 64)])
def test_distance_from_float64_decay_per_channel(heads, vdim):
    case = Channel([300, 33, 64], 2, heads, 128, vdim, torch.bfloat16, heads)
    (out, state), (want, held) = case.run(), case.exact()
    assert off(out, want) <= CLOSE and off(state, held) <= CLOSE


@pytest.mark.parametrize("heads, vdim", [(20, 64), (4, 64)])
def test_distance_from_float64_decay_per_head(heads, vdim):
    """Read-outs as the chain leaves them, and states, from the same unit vectors, strengths and decays."""
    from prefixserve_b200.ops import kernels
    lib, groups, dim, lengths = kernels.lib(), 2, 128, [300, 33, 64]
    g = torch.Generator(device="cuda").manual_seed(heads)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    (ctx, offsets), t, c = step(lengths), sum(lengths), 2 * groups * dim + heads * vdim
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    qkv = torch.cat([unit(rnd(t, 2 * groups, dim)).flatten(1), rnd(t, heads * vdim)], 1)
    bd = torch.cat([torch.rand(t, 2 * heads, generator=g, device="cuda"), rnd(t, 3 * heads)], 1)
    bd[:, heads: 2 * heads] **= 0.1
    proj, held, o = rnd(t, c).bfloat16(), 0.3 * rnd(3, heads * dim * vdim), torch.empty(t, heads, vdim, device="cuda")
    state, chunks = held.clone(), sum(-(-n // 32) for n in lengths)
    records = torch.empty(chunks, heads, lib.psb_delta_chunk_record(dim, vdim), device="cuda")
    kernels.check(lib.psb_delta_chunks(qkv.data_ptr(), bd.data_ptr(), proj.data_ptr(), c, state.data_ptr(), ctx.item_start.data_ptr(), ctx.slots.data_ptr(),
                                       records.data_ptr(), o.data_ptr(), 3, 3, chunks, 1, groups, heads, dim, vdim, 1, 3, held.shape[1], kernels._stream()), "delta_chunks")
    q, k = (qkv[:, a: a + groups * dim].double().view(t, groups, dim).repeat_interleave(heads // groups, 1) for a in (0, groups * dim))
    v, beta, decay = qkv[:, 2 * groups * dim:].double().view(t, heads, vdim), bd[:, :heads].double(), bd[:, heads: 2 * heads].double()
    want, after = [], torch.empty_like(held, dtype=torch.float64)
    for i, n in enumerate(lengths):
        m = held[2 - i].double().view(heads, dim, vdim)
        for j in range(offsets[i], offsets[i] + n):
            m = m * decay[j, :, None, None]
            m = m + k[j, :, :, None] * (beta[j, :, None] * (v[j] - torch.einsum("hd,hdv->hv", k[j], m)))[:, None]
            want.append(torch.einsum("hd,hdv->hv", q[j], m))
        after[2 - i] = m.reshape(-1)
    assert off(o, torch.stack(want)) <= CLOSE and off(state, after) <= CLOSE


@pytest.mark.parametrize("heads, vdim", [(20, 64), (4, 64)])
def test_distance_from_float64_linear_attention(heads, vdim):
    from prefixserve_b200 import ops
    dim, lengths = 128, [300, 33, 64]
    g = torch.Generator(device="cuda").manual_seed(heads)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    (ctx, offsets), t = step(lengths), sum(lengths)
    proj, alpha, held = rnd(t, heads * (2 * dim + vdim)).bfloat16(), torch.sigmoid(rnd(t, heads * dim)) ** (1 / 16), rnd(3, heads * dim * vdim)
    state = held.clone()
    out = ops.linear_attention(proj, alpha, state, ctx, heads=heads, dim=dim, vdim=vdim).view(t, heads, vdim)
    p, a = proj.double(), alpha.double().view(t, heads, dim, 1)
    q, k, v = p[:, : heads * dim].view(t, heads, dim), p[:, heads * dim: 2 * heads * dim].view(t, heads, dim), p[:, 2 * heads * dim:].view(t, heads, vdim)
    want, after = [], torch.empty_like(held, dtype=torch.float64)
    for i, n in enumerate(lengths):
        m = held[2 - i].double().view(heads, dim, vdim)
        for j in range(offsets[i], offsets[i] + n):
            m = a[j] * m + k[j, :, :, None] * v[j, :, None]
            want.append(torch.einsum("hd,hdv->hv", q[j], m) * dim ** -0.5)
        after[2 - i] = m.reshape(-1)
    assert off(out, torch.stack(want)) <= CLOSE and off(state, after) <= CLOSE
