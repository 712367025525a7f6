"""Gated linear attention over long portions, 32 tokens at a time, against the recurrence in float64: portions at and around multiples of
a chunk and of its runs of 16 tokens beside short ones and single tokens, one after the other from carried states, keys and values of
fewer numbers than the kernels' tiles, channels that forget everything and channels that forget nothing, rows and slots that are runs of
wider ones.  (Projections in float32 stay with the kernels that go token by token.)"""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, dim, vdim", [(2, 128, 128), (3, 100, 36), (1, 4, 4), (2, 64, 96)])
def test_long_portions(dtype, heads, dim, vdim):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels, library
    assert kernels.LINEAR_CHUNKED <= 193 and kernels.LINEAR_SHORT == 32
    g = torch.Generator(device="cuda").manual_seed(dim + vdim)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    lengths = [64, 65, 1, 127, 31, 32, 63, 193]
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    offsets = [0]
    for n in lengths:
        offsets.append(offsets[-1] + n)
    ctx = types.SimpleNamespace(item_start=dev(offsets), slots=dev(list(range(len(lengths)))[::-1]), num_items=len(lengths), max_new_tokens=max(lengths))
    held = rnd(len(lengths), heads * dim * vdim + 8)
    state = held[:, : heads * dim * vdim]
    exact, t, width = state.double().clone(), sum(lengths), heads * (2 * dim + vdim)
    for turn in range(2):
        wide = rnd(t, width + 12).to(dtype)
        alpha = torch.sigmoid(rnd(t, heads * dim)) ** (1 / 4)
        alpha[5::9, ::3] = 0.0
        alpha[::4, 1::5] = 1.0
        before = library.launch_counts.copy()
        out = ops.linear_attention(wide[:, : width + 8], alpha, state, ctx, heads=heads, dim=dim, vdim=vdim)
        taken = library.launch_counts - before
        assert taken["linear_attention_chunks"] == (dtype == torch.bfloat16) and taken["linear_attention"] == 1
        for i, n in enumerate(lengths):
            run, slot = slice(offsets[i], offsets[i] + n), len(lengths) - 1 - i
            p = wide[run].double()
            q, k = (p[:, a: a + heads * dim].view(n, heads, dim) for a in (0, heads * dim))
            v, a = p[:, 2 * heads * dim: width].view(n, heads, vdim), alpha[run].double().view(n, heads, dim, 1)
            m, o = exact[slot].view(heads, dim, vdim), []
            for j in range(n):
                m = a[j] * m + k[j, :, :, None] * v[j, :, None]
                o.append(torch.einsum("hd,hdv->hv", q[j], m) * dim ** -0.5)
            exact[slot] = m.reshape(-1)
            # float32 sums of some hundred products of numbers around one
            err = (out[run].double() - torch.stack(o)).abs().max()
            assert err <= 2e-5 * max(1.0, float(torch.stack(o).abs().max())), (turn, i, err)
        assert torch.allclose(state.double(), exact, rtol=1e-5, atol=2e-5), (turn, (state.double() - exact).abs().max())
        assert state.data_ptr() == held.data_ptr()


@pytest.mark.parametrize("what", ["value", "key", "query", "decay"])
def test_a_token_that_is_not_finite_reaches_later_tokens_only(what):
    """As in the recurrence itself: earlier tokens of its chunk, other requests, other heads and (through a value) other columns stay as
    they are."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    heads, dim, vdim, bad = 2, 128, 64, 74   # the eleventh token of a run
    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    ctx = types.SimpleNamespace(item_start=dev([0, 130, 200]), slots=dev([0, 1]), num_items=2, max_new_tokens=130)
    held, proj = rnd(2, heads * dim * vdim), rnd(200, heads * (2 * dim + vdim)).bfloat16()
    alpha = torch.sigmoid(rnd(200, heads * dim)) ** (1 / 4)

    def run(proj, alpha):
        state = held.clone()
        before = library.launch_counts.copy()
        out = ops.linear_attention(proj, alpha, state, ctx, heads=heads, dim=dim, vdim=vdim)
        assert (library.launch_counts - before)["linear_attention_chunks"] == 1
        return out.double().view(200, heads, vdim), state.view(2, heads, dim, vdim)

    clean, _ = run(proj, alpha)
    proj, alpha = proj.clone(), alpha.clone()
    if what == "value":
        proj[bad, 2 * heads * dim + 3] = float("inf")
    elif what == "decay":
        alpha[bad, 5] = float("nan")
    else:
        proj[bad, 5 + (heads * dim if what == "key" else 0)] = float("nan")
    out, state = run(proj, alpha)
    near = lambda a, b: ((a - b).abs() <= 2e-5 * (1 + b.abs().max())).all()   # sums of some hundred products, made again in another order
    assert torch.isfinite(out[:bad]).all() and near(out[:bad], clean[:bad]) and near(out[130:], clean[130:]) and near(out[:, 1:], clean[:, 1:])
    assert torch.isfinite(state[:, 1:]).all() and torch.isfinite(state[1:]).all()
    if what == "value":
        rest = [i for i in range(vdim) if i != 3]
        assert near(out[:, 0, rest], clean[:, 0, rest]) and not torch.isfinite(out[bad:130, 0, 3]).any()
    else:
        assert not torch.isfinite(out[bad, 0]).any()
        if what != "query":
            assert not torch.isfinite(out[129, 0]).any() and not torch.isfinite(state[0, 0, 5]).any()


@pytest.mark.parametrize("lengths, short", [([130, 32, 97], False), ([130, 32, 97, 31], True), ([1, 96], True)])
def test_steps_whose_requests_the_host_holds(lengths, short, monkeypatch):
    """As the engine's contexts: without a short portion the token-by-token kernels are not launched.  Scratch that nobody has written is NaN."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    heads, dim, vdim = 2, 64, 96
    g = torch.Generator(device="cuda").manual_seed(len(lengths))
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    t, offsets = sum(lengths), [0]
    for n in lengths:
        offsets.append(offsets[-1] + n)
    ctx = types.SimpleNamespace(item_start=dev(offsets), slots=dev(list(range(len(lengths)))), num_items=len(lengths), max_new_tokens=max(lengths))
    held, proj, alpha = rnd(len(lengths), heads * dim * vdim), rnd(t, heads * (2 * dim + vdim)).bfloat16(), torch.sigmoid(rnd(t, heads * dim)) ** (1 / 4)

    def run():
        state = held.clone()
        before = library.launch_counts.copy()
        out = ops.linear_attention(proj, alpha, state, ctx, heads=heads, dim=dim, vdim=vdim)
        return out, state, library.launch_counts - before

    out, state, taken = run()
    assert taken["linear_attention"] == 1   # the host does not hold the requests
    ctx.items = [types.SimpleNamespace(start=0, end=n) for n in lengths]
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (lambda x: x.fill_(float("nan")) if x.is_floating_point() else x)(empty(*a, **k)))
    again, state_again, taken = run()
    assert taken["linear_attention_chunks"] == 1 and taken["linear_attention"] == short
    assert torch.equal(out, again) and torch.equal(state, state_again)


@pytest.mark.parametrize("tokens", [100, 600])
def test_no_further_from_float64_than_token_by_token(tokens, monkeypatch):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels
    heads, dim, vdim = 8, 128, 128
    g = torch.Generator(device="cuda").manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    ctx = types.SimpleNamespace(item_start=dev([0, tokens]), slots=dev([0]), num_items=1, max_new_tokens=tokens)
    held, proj, alpha = rnd(1, heads * dim * vdim), rnd(tokens, heads * (2 * dim + vdim)).bfloat16(), torch.sigmoid(rnd(tokens, heads * dim)) ** (1 / 16)
    p, m, want = proj.double(), held[0].double().view(heads, dim, vdim), []
    q, k = (p[:, a: a + heads * dim].view(tokens, heads, dim) for a in (0, heads * dim))
    v, a = p[:, 2 * heads * dim:].view(tokens, heads, vdim), alpha.double().view(tokens, heads, dim, 1)
    for j in range(tokens):
        m = a[j] * m + k[j, :, :, None] * v[j, :, None]
        want.append(torch.einsum("hd,hdv->hv", q[j], m) * dim ** -0.5)
    want, off = torch.stack(want), {}
    for which, line in (("chunks", 96), ("tokens", 1 << 30)):
        monkeypatch.setattr(kernels, "LINEAR_CHUNKED", line)
        state = held.clone()
        out = ops.linear_attention(proj, alpha, state, ctx, heads=heads, dim=dim, vdim=vdim)
        off[which] = [float((x.double() - e).norm() / e.norm()) for x, e in ((out, want), (state.view(heads, dim, vdim), m))]
    # (the distances are sums of millions of roundings and hold to a few hundredths; 0.94 and 0.84 of the other kernels')
    assert off["chunks"][0] <= off["tokens"][0] and off["chunks"][1] <= off["tokens"][1], off


@pytest.mark.parametrize("heads", [1, 40])   # a run of columns a block, and two
def test_read_outs_of_an_infinite_state(heads):
    """As in the recurrence: a query reads infinity of that channel's sign from the column, and the other columns as they are."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    n, dim, vdim = 100, 128, 64
    g = torch.Generator(device="cuda").manual_seed(heads)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    ctx = types.SimpleNamespace(item_start=dev([0, n]), slots=dev([0]), num_items=1, max_new_tokens=n)
    held, proj, alpha = rnd(1, heads, dim, vdim), rnd(n, heads * (2 * dim + vdim)).bfloat16(), 0.5 + 0.5 * torch.sigmoid(rnd(n, heads * dim))

    def run(held):
        state = held.clone().view(1, -1)
        before = library.launch_counts.copy()
        out = ops.linear_attention(proj, alpha, state, ctx, heads=heads, dim=dim, vdim=vdim)
        assert (library.launch_counts - before)["linear_attention_chunks"] == 1
        return out.view(n, heads, vdim), state.view(heads, dim, vdim)

    clean, state = run(held)
    held[0, 0, 77, 21], held[0, 0, 3, 40] = float("inf"), float("-inf")
    out, after = run(held)
    query = proj[:, : heads * dim].float().view(n, heads, dim)
    rest = [c for c in range(vdim) if c not in (21, 40)]
    for channel, column, sign in ((77, 21, 1.0), (3, 40, -1.0)):
        assert torch.equal(out[:, 0, column], sign * torch.sign(query[:, 0, channel]) * float("inf")) and after[0, channel, column] == sign * float("inf")
    assert torch.equal(out[:, 0, rest], clean[:, 0, rest]) and torch.equal(out[:, 1:], clean[:, 1:])
    finite = torch.isfinite(after)
    assert int((~finite).sum()) == 2 and torch.equal(after[finite], state[finite])


def test_more_chunks_than_a_grid_has_rows():
    """A portion of more than 65,535 chunks, against the same tokens in two portions, one after the other."""
    from prefixserve_b200 import ops
    n, first, dim, vdim = 32 * 65536 + 1, 32 * 40000, 4, 4
    g = torch.Generator(device="cuda").manual_seed(6)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    held, proj, alpha = rnd(1, dim * vdim), rnd(n, 2 * dim + vdim).bfloat16(), torch.sigmoid(rnd(n, dim)) ** 0.25

    def run(state, a, b):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        ctx = types.SimpleNamespace(item_start=dev([0, b - a]), slots=dev([0]), num_items=1, max_new_tokens=b - a, items=[types.SimpleNamespace(start=a, end=b)])
        return ops.linear_attention(proj[a:b], alpha[a:b], state, ctx, heads=1, dim=dim, vdim=vdim)

    whole, parts = held.clone(), held.clone()
    out = run(whole, 0, n)
    assert torch.equal(out, torch.cat([run(parts, 0, first), run(parts, first, n)])) and torch.equal(whole, parts)
