"""Routed experts with a few rows each, whose matrices are streamed through mma.sync by blocks that take equal runs of (expert, eight
rows, 32 columns): experts without rows, with one, with exactly eight and with more than one pass of eight, sums that end inside a
warp's first turn and behind several, columns that end inside a slab, an odd number of experts, fewer units than blocks and more."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h, ff", [(8, 24), (72, 40), (520, 136), (1032, 520), (4104, 64), (64, 12296), (256, 1024)])
@pytest.mark.parametrize("glu", [None, "silu"])
def test_few_rows(h, ff, glu):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    g = torch.Generator(device="cuda").manual_seed(h + ff)
    rnd = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(torch.bfloat16)
    rows = [0, 1, 8, 0, 17, 3, 9]
    experts, t = len(rows), sum(rows) // 2
    of = torch.tensor([e for e, n in enumerate(rows) for _ in range(n)], dtype=torch.int32)
    chosen = of[torch.randperm(2 * t, generator=torch.Generator().manual_seed(ff))].view(t, 2).cuda().contiguous()
    weight = torch.rand(t, 2, generator=g, device="cuda")
    x, up, down = rnd(t, h), rnd(experts, ff * (2 if glu else 1), h, std=h ** -0.5), rnd(experts, h, ff, std=ff ** -0.5)
    before = library.launch_counts.copy()
    out = ops.moe_experts(x, chosen, weight, up, down, activation=None, glu=glu, out_dtype=torch.float32)
    assert (library.launch_counts - before)["moe_gemm"] == 2
    mid = torch.einsum("tk,tpnk->tpn", x.double(), up.double()[chosen.long()])
    spread = 2.0 ** -8 * mid.abs()  # both products' operands are bfloat16: the first one's results are rounded (half a place in 2^8) ...
    if glu:
        gate, value = mid.chunk(2, -1)
        mid = torch.nn.functional.silu(gate) * value
        # ... and with a gate (slope at most 1.1) both of its arguments, and its result again
        a, b = spread.chunk(2, -1)
        spread = 1.1 * a * value.abs() + b * torch.nn.functional.silu(gate).abs() + 2.0 ** -8 * mid.abs() + 1.1 * a * b
    picked = down.double()[chosen.long()]
    want = torch.einsum("tp,tpn,tphn->th", weight.double(), mid, picked)
    bound = torch.einsum("tp,tpn,tphn->th", weight.double(), spread + 1e-6 * (1 + mid.abs()), picked.abs()) + 1e-6
    assert ((out.double() - want).abs() <= bound).all(), ((out.double() - want).abs() / bound).max()


@pytest.mark.parametrize("ff", [4096, 12296])
def test_sums_are_rounded_not_cut_off(ff):
    """Sums of positive terms: what an accumulator cuts off at every step would add up to a bias.  The first product picks a column,
    so that the second one's operands are exact."""
    from prefixserve_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(ff)
    h, experts, t = 256, 6, 20
    x = torch.zeros(t, h, device="cuda", dtype=torch.bfloat16)
    x[:, 0] = 1.0
    up = torch.rand(experts, ff, h, generator=g, device="cuda").to(torch.bfloat16)
    down = torch.rand(experts, h, ff, generator=g, device="cuda").to(torch.bfloat16)
    chosen = torch.randint(experts, (t, 1), generator=g, device="cuda").to(torch.int32)
    out = ops.moe_experts(x, chosen, torch.ones(t, 1, device="cuda"), up, down, activation=None, out_dtype=torch.float32)
    e = chosen[:, 0].long()
    want = torch.einsum("tp,thp->th", up[e, :, 0].double(), down[e].double())
    off = out.double() / want - 1
    # float32 sums rounded to nearest err on both sides; an instruction cuts less than 2^-23 of its own 16 terms off
    assert off.mean().abs() <= 2.0 ** -23, off.mean()
    assert off.abs().max() <= (ff / 128 + 8) * 2.0 ** -24, off.abs().max()
