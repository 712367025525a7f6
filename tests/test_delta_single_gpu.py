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
