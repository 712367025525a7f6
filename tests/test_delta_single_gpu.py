"""The delta rules' kernel for steps of single tokens: against the recurrence in float64, and beside the kernels that take any portion.

Bound: a head's read-out is a sum of up to 128 products of float32 numbers over a state of such sums: 64 half units of the last place at most on the
numbers' scale, 4e-6 of the largest; the kernels were measured at 1 to 3e-7 of it in the 2-norm.  bfloat16 results add their own rounding, 2^-8 of a number."""

import types

import pytest
import torch

from prefixserve_b200 import ops
from prefixserve_b200.ops import library

pytestmark = pytest.mark.gpu

EPS = 1e-6


def _silu(x):
    return x / (1 + torch.exp(-x))


def _oracle(proj, ba, decay, beta_at, taps, a_log, dt_bias, gain, state, positions, slots, groups, heads, dim, vdim, gated):
    """(result, state) in float64, a token a request."""
    state = state.clone()
    k, c = taps.shape[1], 2 * groups * dim + heads * vdim
    out = []
    for t, (p, slot) in enumerate(zip(positions, slots)):
        kept = state[slot][: (k - 1) * c].view(k - 1, c)
        rows = torch.cat([kept, proj[t: t + 1, :c]])
        seen = rows.clone()
        seen[: max(0, k - 1 - p)] = 0
        x = _silu((seen * taps.t()).sum(0))
        q, key, v = x[: groups * dim].view(groups, dim), x[groups * dim: 2 * groups * dim].view(groups, dim), x[2 * groups * dim:].view(heads, vdim)
        q = q / torch.sqrt((q * q).sum(1, keepdim=True) + 1e-6) / dim ** 0.5
        key = key / torch.sqrt((key * key).sum(1, keepdim=True) + 1e-6)
        S = state[slot][(k - 1) * c:].view(heads, dim, vdim)
        o = torch.empty(heads, vdim, dtype=torch.float64, device=proj.device)
        for h in range(heads):
            g = h // (heads // groups)
            beta = torch.sigmoid(ba[t, h] if gated else proj[t, beta_at + h])
            if gated:
                S[h] *= torch.exp(-torch.exp(a_log[h]) * torch.nn.functional.softplus(ba[t, heads + h] + dt_bias[h]))
            else:
                S[h] *= decay[t].view(heads, dim)[h][:, None]
            S[h] += torch.outer(key[g], beta * (v[h] - S[h].t() @ key[g]))
            o[h] = S[h].t() @ q[g]
        if gated:
            o = o / torch.sqrt((o * o).mean(1, keepdim=True) + EPS) * gain * _silu(proj[t, c: c + heads * vdim].view(heads, vdim))
        state[slot][: (k - 1) * c] = rows[1:].reshape(-1)
        out.append(o)
    return torch.stack(out), state


@pytest.mark.parametrize("groups,heads,dim,vdim,k,dtype", [(8, 16, 128, 128, 4, torch.bfloat16), (2, 4, 16, 24, 4, torch.float32), (1, 8, 128, 4, 2, torch.float32),
                                                           (3, 3, 100, 128, 1, torch.bfloat16), (2, 6, 7, 60, 16, torch.float32), (1, 1, 128, 128, 3, torch.bfloat16)])
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("requests", [1, 5])
def test_single_tokens(groups, heads, dim, vdim, k, dtype, gated, requests):
    gen = torch.Generator(device="cuda").manual_seed(groups * 100 + dim + requests)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    c = 2 * groups * dim + heads * vdim
    if (k - 1) * c % 4:
        pytest.skip("the slots' states do not start at a multiple of four numbers: another kernel's")
    beta_at = c + 3
    proj = rand(requests, c + heads * vdim if gated else beta_at + heads).to(dtype)
    ba, decay = rand(requests, 2 * heads), torch.sigmoid(rand(requests, heads * dim) + 2)
    taps, a_log, dt_bias, gain = rand(c, k) * 0.5, rand(heads) * 0.3, rand(heads), rand(vdim)
    state0 = rand(requests + 2, (k - 1) * c + heads * dim * vdim)
    positions = [0, 1, 2, 40, 700][:requests] if requests > 1 else [3]
    slots = [requests - i for i in range(requests)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")

    def call(longest):
        ctx = types.SimpleNamespace(positions=i32(positions), token_item=i32(list(range(requests))), item_start=i32(list(range(requests + 1))), slots=i32(slots),
                                    num_items=requests, max_new_tokens=longest)
        state = state0.clone()
        before = library.launch_counts.copy()
        if gated:
            out = ops.delta_rule(proj, ba, taps, a_log, dt_bias, gain, state, ctx, groups=groups, heads=heads, dim=dim, vdim=vdim, eps=EPS)
        else:
            out = ops.channel_delta_rule(proj, beta_at, decay, taps, state, ctx, groups=groups, heads=heads, dim=dim, vdim=vdim)
        return out.view(requests, heads, vdim), state, library.launch_counts - before

    d = lambda x: x.double()
    want, want_state = _oracle(d(proj), d(ba), d(decay), beta_at, d(taps), d(a_log), d(dt_bias), d(gain), d(state0), positions, slots, groups, heads, dim, vdim, gated)
    out, state, taken = call(1)
    assert taken["delta_single"] == 1 and sum(taken.values()) == 1
    other, other_state, taken = call(2)  # a step that is said to hold longer portions
    assert taken["delta_single"] == 0
    far = lambda x, y: float((x.double() - y).norm() / y.norm())
    assert far(state, want_state) < 4e-6 and far(state, want_state) < 1.5 * far(other_state, want_state) + 2e-7
    rounding = 2.0 ** -8 if gated and dtype == torch.bfloat16 else 0.0
    assert float((out.double() - want).abs().max()) <= (4e-6 + rounding) * float(want.abs().max())
    assert far(out, want) < 1.5 * far(other, want) + 2e-7
    untouched = [s for s in range(requests + 2) if s not in slots]
    assert torch.equal(state[untouched], state0[untouched])


@pytest.mark.parametrize("gated", [True, False])
def test_a_wait_that_gives_up_leaves_everything_as_it_was(gated):
    """The wait for a head's state gives up at once: its code stands in the word handed in, and neither state, inputs nor result are touched."""
    groups, heads, dim, vdim, k, requests = 2, 4, 64, 32, 4, 3
    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    c = 2 * groups * dim + heads * vdim
    proj = rand(requests, c + heads * vdim if gated else c + heads)
    ba, decay, taps, a_log, dt_bias, gain = rand(requests, 2 * heads), torch.rand(requests, heads * dim, device="cuda"), rand(c, k), rand(heads), rand(heads), rand(vdim)
    state, out, word = rand(requests, (k - 1) * c + heads * dim * vdim), rand(requests, heads * vdim), i32([0])
    positions, item_start, slots = i32([0, 5, 700]), i32([0, 1, 2, 3]), i32([2, 0, 1])
    of = lambda x, there: x.data_ptr() if there else None

    def call(state, out, word):
        library.check(library.lib().psb_delta_single(
            proj.data_ptr(), 0, proj.shape[1], 0 if gated else c, of(ba, gated), of(decay, not gated), taps.data_ptr(), of(a_log, gated), of(dt_bias, gated),
            state.data_ptr(), positions.data_ptr(), item_start.data_ptr(), slots.data_ptr(), of(gain, gated), out.data_ptr(), requests, groups, heads, dim, vdim, k,
            requests, state.shape[1], EPS, word, library.stream_handle()), "delta_single")

    state2, out2 = state.clone(), out.clone()
    call(state2, out2, word.data_ptr())
    assert word.item() == 1 and torch.equal(state2, state) and torch.equal(out2, out)
    assert library.tcgen05_status() == 0  # (the word of the kernel itself is another)
    call(state2, out2, None)
    changed = (state2 != state).view(requests, -1)
    assert bool(changed.any(1).all()) and not torch.equal(out2, out) and library.tcgen05_status() == 0


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("groups,heads,dim,vdim,k", [(2, 4, 64, 32, 4), (1, 2, 128, 128, 4), (1, 1, 9, 4, 1)])
def test_numbers_that_are_not_finite(gated, groups, heads, dim, vdim, k):
    """Infinite and NaN projections, states, inputs and gates, and decays of 0, one kind a request: finite numbers, infinities and NaN stand where the kernels that
    take any portion leave them, the finite ones as close as ever, and a request beside them is untouched by them."""
    gen = torch.Generator(device="cuda").manual_seed(dim + gated)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    c = 2 * groups * dim + heads * vdim
    inf, nan, n = float("inf"), float("nan"), 14
    proj = rand(n, c + heads * vdim if gated else c + heads)
    ba, decay = rand(n, 2 * heads), torch.sigmoid(rand(n, heads * dim) + 2)
    taps, a_log, dt_bias, gain = rand(c, k) * 0.5, rand(heads) * 0.3, rand(heads), rand(vdim)
    state = rand(n, (k - 1) * c + heads * dim * vdim)
    S = state[:, (k - 1) * c:].view(n, heads, dim, vdim)
    proj[0, 1], proj[1, groups * dim], proj[2, 2 * groups * dim + 1], proj[3, 2 * groups * dim] = nan, inf, -inf, 1e30   # query, key, values
    S[4, 0, 0, 1], S[5, -1, 3, 2], S[6, 0, 1, 0], S[7, 0, 2, 3] = inf, -inf, nan, 3e38  # (a whole column of the last overflows or not by the order of its sum)
    if k > 1:
        state[8, 0], state[9, 2 * groups * dim] = nan, inf                                                              # inputs kept from before
    if gated:
        ba[10, 0], ba[11, heads], ba[12, heads] = inf, 3e4, nan                                                         # strength; a decay of 0
        proj[13, c] = nan                                                                                               # the output gate
        S[11, 0, 0, 0] = inf                                                                                            # 0 times that
    else:
        proj[10, c] = -inf
        decay[11], decay[12, 1], decay[13, 0] = 0.0, nan, inf
        S[11, 0, 0, 0] = inf
    positions, token_item, starts, slots = i32([5] * n), i32(list(range(n))), i32(list(range(n + 1))), i32(list(range(n)))

    def call(longest):
        ctx = types.SimpleNamespace(positions=positions, token_item=token_item, item_start=starts, slots=slots, num_items=n, max_new_tokens=longest)
        mine = state.clone()
        if gated:
            out = ops.delta_rule(proj, ba, taps, a_log, dt_bias, gain, mine, ctx, groups=groups, heads=heads, dim=dim, vdim=vdim, eps=EPS)
        else:
            out = ops.channel_delta_rule(proj, c, decay, taps, mine, ctx, groups=groups, heads=heads, dim=dim, vdim=vdim)
        return out.view(n, -1), mine

    (out, mine), (other, theirs) = call(1), call(2)
    for got, want in ((out, other), (mine, theirs)):
        for r in range(n):
            assert torch.equal(got[r].isnan(), want[r].isnan()), r
            assert torch.equal(got[r].nan_to_num(0.0, 7.0, -7.0)[got[r].isinf()], want[r].nan_to_num(0.0, 7.0, -7.0)[want[r].isinf()]), r
            fine = got[r].isfinite()
            if bool(fine.any()):
                far = (got[r][fine].double() - want[r][fine].double()).abs().max()
                assert float(far) <= 8e-6 * float(want[r][fine].double().abs().max()), r
