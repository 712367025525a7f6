"""Prompt portions on the kernel of 128-row tiles where its launch is not the plain one (short portions behind long contexts, row groups of a second round halved):
which kernel attends for them, and how far the results are from float64.

Bound: weights and results are rounded to bfloat16, each by at most 2^-9 of a number, independently of one another: sqrt(2) 2^-9 of the results in the 2-norm.
(A key too many or too few in every row changes results over 4,000 keys by 1 / sqrt(4,000), six times that.)  A short portion's results are besides
no further from float64 than those of the kernel that would take them otherwise; 1 % is what the order of float32 sums and a few
hundred rows' roundings may differ by."""

import pytest
import torch

from prefixserve_b200 import ops
from prefixserve_b200.engine import StepItem  # noqa: F401  (the engine's package loads)
from prefixserve_b200.ops import library, tensorcore
from prefixserve_b200.parts.base import ItemView, StepContext

pytestmark = pytest.mark.gpu


def _step(d, hq, hkv, portions):
    page, gen = 16, torch.Generator(device="cuda").manual_seed(d + len(portions))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    starts, views = [0], []
    for i, (n, held) in enumerate(portions):
        views.append(ItemView(slot=i, start=held, end=held + n, first_token=starts[-1]))
        starts.append(starts[-1] + n)
    width = max(-(-(n + held) // page) for n, held in portions)
    table = torch.randperm(len(portions) * width, generator=gen, device="cuda").to(torch.int32).view(len(portions), width)
    ctx = StepContext(
        num_tokens=starts[-1], num_items=len(portions), compute_dtype=torch.bfloat16, device=torch.device("cuda"), items=views,
        token_ids=i32([0] * starts[-1]), positions=i32([p for n, held in portions for p in range(held, held + n)]),
        token_item=i32([i for i, (n, _) in enumerate(portions) for _ in range(n)]), item_start=i32(starts), kv_len=i32([n + held for n, held in portions]),
        slots=i32(list(range(len(portions)))), block_tables={0: table}, max_new_tokens=max(n for n, _ in portions),
        max_kv_len=max(n + held for n, held in portions), all_decode=False)
    q = torch.randn(starts[-1], hq, d, generator=gen, device="cuda").to(torch.bfloat16)
    kv = torch.randn(len(portions) * width, 2, hkv, page, d, generator=gen, device="cuda").to(torch.bfloat16)
    return ctx, table, q, kv


def _far(out, ctx, table, q, kv, window):
    """Distance from attention in float64, relative, in the 2-norm."""
    off = of = 0.0
    out = out.view_as(q).double()
    for i, it in enumerate(ctx.items):
        rows = kv[table[i].long()]
        keys, values = (rows[:, p].transpose(1, 2).reshape(-1, rows.shape[2], rows.shape[4])[: it.end].double() for p in (0, 1))
        at, own = torch.arange(it.end, device="cuda")[None, :], torch.arange(it.start, it.end, device="cuda")[:, None]
        seen = (at <= own) & (at > own - (window or it.end + 1))
        here = slice(it.first_token, it.first_token + it.end - it.start)
        for h in range(q.shape[1]):
            g = h // (q.shape[1] // keys.shape[1])
            s = (q[here, h].double() @ keys[:, g].t() * q.shape[2] ** -0.5).masked_fill(~seen, float("-inf"))
            want = torch.softmax(s, dim=1) @ values[:, g]
            off, of = off + float((out[here, h] - want).pow(2).sum()), of + float(want.pow(2).sum())
    return (off / of) ** 0.5


ROUNDINGS = 2 ** 0.5 * 2.0 ** -9


@pytest.mark.parametrize("d,hq,hkv,window,portions,taken", [
    (64, 32, 8, None, [(31, 2000)], True), (64, 32, 8, None, [(2, 1407)], True), (64, 32, 8, None, [(2, 1406)], False),       # 12 blocks of keys: three ranges
    (64, 8, 1, None, [(9, 3000), (63, 1500), (1, 400)], True), (64, 32, 8, None, [(9, 1500)] * 2, False),                      # 64 CTAs: two ranges
    (128, 32, 8, None, [(2, 510)], True), (128, 32, 8, None, [(2, 509)], False),                                               # 512 keys
    (128, 32, 8, None, [(63, 449), (1, 700), (5, 100)], True), (128, 32, 8, None, [(63, 448)], False),                         # 512 keys; beside a decoded token
    (128, 32, 8, None, [(9, 1500)] * 4, True), (128, 32, 8, None, [(9, 1500)] * 5, False),                                     # 128 and 160 CTAs
    (128, 32, 32, None, [(8, 600)] * 3, True), (128, 16, 1, None, [(24, 1000)], True),
    (128, 8, 8, 300, [(20, 3000)], False), (128, 8, 4, 500, [(20, 3000), (1, 2000)], True), (128, 6, 1, None, [(3, 4000)], True)])
def test_short_portions(monkeypatch, d, hq, hkv, window, portions, taken):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the numbers of CTAs are for 148 SMs")
    ctx, table, q, kv = _step(d, hq, hkv, portions)

    def call():
        ctx.extras.clear()  # (the plan a step keeps for its layers)
        before = library.launch_counts.copy()
        out = ops.attention(q, kv, table, ctx.positions, ctx.token_item, window=window, ctx=ctx)
        return out, library.launch_counts - before

    out, counts = call()
    assert counts["attention_prefill_tcgen05"] == taken and counts["attention_prefill"] == (not taken)
    far = _far(out, ctx, table, q, kv, window)
    assert library.tcgen05_status() == 0
    assert far <= ROUNDINGS
    if taken:
        monkeypatch.setattr(tensorcore, "TCGEN05_SHORT_MIN_KEYS", 1 << 30)
        other, counts = call()
        assert counts["attention_prefill"] == 1
        assert far <= 1.01 * _far(other, ctx, table, q, kv, window)


@pytest.mark.parametrize("d,portions,groups,whole", [(64, [(640, 300), (512, 40)], 5, 4), (128, [(641, 300), (513, 40)], 6, 4), (128, [(1152, 7)], 5, 4), (64, [(700, 0), (560, 90)], 6, 6),
                                                     (64, [(1025, 500), (1, 900)], 5, 4), (128, [(2048, 0)], 8, 8)])
def test_row_groups_of_a_second_round(d, portions, groups, whole):
    hq, hkv, sms = 32, 8, torch.cuda.get_device_properties(0).multi_processor_count
    if sms != 148:
        pytest.skip("the numbers of groups are for 148 SMs")
    plan = tensorcore._attention_plan([n for n, _ in portions], [n + held for n, held in portions], 0, hq // hkv, hkv, d, 16, sms, None)
    assert plan["tcgen05"] and (plan["pairs"], plan["whole"]) == (groups, whole)
    ctx, table, q, kv = _step(d, hq, hkv, portions)
    out = ops.attention(q, kv, table, ctx.positions, ctx.token_item, ctx=ctx)
    assert library.tcgen05_status() == 0
    assert _far(out, ctx, table, q, kv, None) <= ROUNDINGS
