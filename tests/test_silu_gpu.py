"""The SiLU without a division in the passes around the delta rules (csrc/kernels/delta_common.cuh), as the results of those passes hold it.

Bound: exp is good to 2 units of the last place (CUDA's own statement for float32), of which the quotient's denominator keeps no more; adding one and the quotient round
half a unit each: 3 units from float64.  From the division itself a corrected quotient differs by a unit at most, and that seldom (it rounds alike but for cases within
2^-47 of the middle between two numbers; 1 in 1,000 is far above)."""

import pytest
import torch

from prefixserve_b200.ops import library

pytestmark = pytest.mark.gpu
GROUPS, HEADS, DIM, VDIM = 4, 8, 32, 64


def _units(got, want):
    """Differences in units of the last place of ``want`` (float64)."""
    return (got.double() - want).abs() / torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -126))) - 23)


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def _prepared(proj):
    """The value channels of the wide preparing kernel with one tap of 1: silu of the projection."""
    t, c = proj.shape
    slot = HEADS * DIM * VDIM
    qkv, bd = torch.empty(t, c, device="cuda"), torch.empty(t, 5 * HEADS, device="cuda")
    ba, zeros = torch.zeros(t, 2 * HEADS, device="cuda"), torch.zeros(max(HEADS, slot), device="cuda")
    positions, items, starts, slots = torch.arange(t, dtype=torch.int32, device="cuda"), torch.zeros(t, dtype=torch.int32, device="cuda"), _i32([0, t]), _i32([0])
    taps = torch.ones(c, 1, device="cuda")
    library.check(library.lib().psb_delta_prepare(
        proj.data_ptr(), 0, c, 0, ba.data_ptr(), None, taps.data_ptr(), zeros.data_ptr(), zeros.data_ptr(), zeros.data_ptr(), positions.data_ptr(), items.data_ptr(),
        starts.data_ptr(), slots.data_ptr(), qkv.data_ptr(), bd.data_ptr(), t, GROUPS, HEADS, DIM, VDIM, 1, 1, slot, 0, library.stream_handle()), "delta_prepare")
    return qkv[:, 2 * GROUPS * DIM:]


def _finished(gate):
    """The finishing kernel over read-outs of 1 with a gain of 1: silu of the gate, times what makes a mean square of 1 one (1 itself)."""
    t, c = gate.shape[0], 2 * GROUPS * DIM + HEADS * VDIM
    proj = torch.cat([torch.zeros(t, c, device="cuda"), gate], dim=1).contiguous()
    out, gain = torch.empty(t, HEADS * VDIM, device="cuda"), torch.ones(VDIM, device="cuda")
    o = torch.ones(t, HEADS, VDIM, device="cuda")
    library.check(library.lib().psb_delta_finish(o.data_ptr(), proj.data_ptr(), 0, gain.data_ptr(), out.data_ptr(), t, GROUPS, HEADS, DIM, VDIM, 0.0,
                                                 library.stream_handle()), "delta_finish")
    return out


@pytest.mark.parametrize("through", ["prepare", "finish"])
def test_silu_of_any_size(through):
    t, gen = 203, torch.Generator(device="cuda").manual_seed(3)
    width = HEADS * VDIM
    x = (torch.rand(t, width, generator=gen, device="cuda") * 2 - 1) * torch.tensor([1e-3, 1.0, 20.0, 79.9], device="cuda").repeat(width // 4)
    far = x.clone()
    far[7, 5], far[100], far[150, 3], far[151, ::2] = 80.5, 87.0, -81.0, -200.0  # one number, a whole token, below, where the exponential overflows
    far[160, 1], far[160, 2], far[160, 3] = float("inf"), float("-inf"), float("nan")

    def call(values):
        if through == "finish":
            return _finished(values)
        return _prepared(torch.cat([torch.ones(t, 2 * GROUPS * DIM, device="cuda"), values], dim=1).contiguous())

    got, beside = call(x), call(far)
    near = far == x
    assert torch.equal(got[near], beside[near])  # no number's result depends on its neighbours'
    divided = far / (1 + torch.exp(-far))
    beyond = ~near
    assert torch.equal(beside[beyond].nan_to_num(nan=7.0), divided[beyond].nan_to_num(nan=7.0))  # the division itself
    assert float((got != (x / (1 + torch.exp(-x)))).float().mean()) < 1e-3
    want = x.double() / (1 + torch.exp(-x.double()))
    off = _units(got, want)
    assert float(off.max()) <= 3.0 and float(off.pow(2).mean().sqrt()) < 0.6
