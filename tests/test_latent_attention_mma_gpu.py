"""Single tokens' latent attention on the tensor cores (rows of 512 + 64 numbers, heads in groups of 16 and 32) against the
same sums in float64: every number of heads a block takes, windows, keys split among blocks and not, the borders of its key
tiles and of pages, sinks and gates, pages that are not there."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu

RANK, ROT = 512, 64


def case(lengths, heads, page, seed, dead=()):
    g = torch.Generator().manual_seed(seed)
    need = [-(-n // page) for n in lengths]
    ids = torch.randperm(sum(need), generator=g).tolist()
    table = torch.full((len(lengths), max(need)), -1, dtype=torch.int32)
    cache = torch.full((sum(need), 1, 1, page, RANK + ROT), float("nan"), dtype=torch.bfloat16)
    rows = [torch.randn(n, RANK + ROT, generator=g).bfloat16() for n in lengths]
    for i, r in enumerate(rows):
        for j in range(need[i]):
            table[i, j] = pid = ids.pop()
            cache[pid, 0, 0, : len(r[j * page: (j + 1) * page])] = r[j * page: (j + 1) * page]
    for i, j in dead:
        table[i, j] = -1
    q = torch.randn(len(lengths), heads, RANK + ROT, generator=g) * 0.6
    positions = torch.tensor([n - 1 for n in lengths], dtype=torch.int32)
    items = [types.SimpleNamespace(start=n - 1, end=n, first_token=i) for i, n in enumerate(lengths)]
    return q, cache, table, rows, positions, items


def expected(q, rows, i, n, window, scale, sink, page, dead):
    keys = rows[i].double()
    s = q[i].double() @ keys.t() * scale
    seen = torch.ones(n, dtype=torch.bool)
    if window:
        seen[: max(0, n - window)] = False
    for a, j in dead:
        if a == i:
            seen[j * page: (j + 1) * page] = False
    s = s.masked_fill(~seen, float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None]], 1)
    return torch.softmax(s, 1)[:, :n] @ keys[:, :RANK]


@pytest.mark.parametrize("heads,window,page,with_sink,with_gate,dead", [
    (16, None, 16, True, False, ()), (32, None, 16, False, True, ()), (48, 300, 16, True, True, ()), (64, 33, 32, False, False, ()),
    (32, 64, 5, True, False, ()), (16, 1, 16, False, True, ()), (32, None, 16, False, False, ((2, 3), (4, 0))),
])
def test_single_tokens(heads, window, page, with_sink, with_gate, dead):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels
    lengths = [1, 31, 65, 64, 129, 700, 32, 1500]
    q, cache, table, rows, positions, items = case(lengths, heads, page, heads + page, dead)
    g = torch.Generator().manual_seed(9)
    sink = torch.randn(heads, generator=g) + 1.0 if with_sink else None
    gate = torch.rand(len(lengths), heads, generator=g) if with_gate else None
    assert kernels.lib().psb_latent_attention_mma_heads(RANK, ROT, heads) == (32 if heads % 32 == 0 else 16)
    item = torch.arange(len(lengths), dtype=torch.int32).cuda()
    dev = lambda x: None if x is None else x.cuda()
    got = {}
    for hint in (0, 1500, 60000):   # one block a token, a few, many
        out = ops.latent_attention(q.cuda(), cache.cuda(), table.cuda(), positions.cuda(), item, dev(gate), rank=RANK, page_size=page,
                                   window=window, scale=0.07, out_dtype=torch.bfloat16, items=items, key_hint=hint, sink=dev(sink))
        got[hint] = out.cpu().double()
    for i, n in enumerate(lengths):
        want = expected(q, rows, i, n, window, 0.07, sink, page, dead)
        if gate is not None:
            want = want * gate[i].double()[:, None]
        for hint, out in got.items():
            # the result is rounded to bfloat16 (2^-9 of a value); scores, weights and sums are float32
            assert ((out[i] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all(), (i, n, hint, (out[i] - want).abs().max())


def test_other_sizes_and_types_keep_their_kernels():
    from prefixserve_b200.ops import kernels
    lib = kernels.lib()
    assert [lib.psb_latent_attention_mma_heads(*s) for s in ((512, 64, 8), (512, 64, 20), (256, 64, 32), (512, 32, 16), (512, 64, 96))] == [0, 0, 0, 0, 32]


@pytest.mark.parametrize("heads", [16, 32])
def test_a_row_that_scores_minus_infinity_drops_out(heads):
    """A cached row with an infinite rotated number, against queries whose number there is one bfloat16 term (the others are 0); a row
    that scores +inf, against other heads, makes their result NaN and nobody else's."""
    from prefixserve_b200 import ops
    lengths, page = [70, 200], 16
    q, cache, table, rows, positions, items = case(lengths, heads, page, 1)
    q[:, :, RANK + 3] = 1.0
    q[1, 0, RANK + 3] = -1.0
    for i, key in ((0, 5), (0, 69), (1, 150)):
        cache[table[i, key // page], 0, 0, key % page, RANK + 3] = rows[i][key, RANK + 3] = float("-inf")
    for hint in (0, 60000):
        out = ops.latent_attention(q.cuda(), cache.cuda(), table.cuda(), positions.cuda(), torch.arange(2, dtype=torch.int32).cuda(), None, rank=RANK,
                                   page_size=page, window=None, scale=0.07, out_dtype=torch.bfloat16, items=items, key_hint=hint).cpu().double()
        for i, n in enumerate(lengths):
            want = expected(q, rows, i, n, None, 0.07, None, page, ())
            for h in range(heads):
                if (i, h) == (1, 0):
                    assert not torch.isfinite(out[i, h]).any()
                else:   # as in test_single_tokens
                    assert ((out[i, h] - want[h]).abs() <= 2.0 ** -8 * want[h].abs() + 1e-4).all(), (hint, i, h)


def test_sums_are_rounded_not_cut_off():
    """Positive numbers, where what an accumulator cuts off at every step would add up to a bias: the shares that the blocks leave,
    before they are joined and rounded to bfloat16."""
    from prefixserve_b200.ops import kernels
    heads, n, page, splits = 32, 3000, 16, 2
    q, cache, table, rows, positions, _ = case([n], heads, page, 3)
    q, cache, rows = q.abs() * 0.3, cache.abs(), [r.abs() for r in rows]
    dev = [x.cuda() for x in (q, cache, table, positions, torch.zeros(1, dtype=torch.int32))]
    out = torch.empty(1, heads, RANK, dtype=torch.bfloat16, device="cuda")
    partial = torch.zeros(1, heads, splits, RANK + 2, device="cuda")
    ptr = [x.data_ptr() for x in dev]
    kernels.check(kernels.lib().psb_latent_attention_mma(ptr[0], ptr[1], ptr[2], table.shape[1], ptr[3], ptr[4], None, out.data_ptr(), 1, heads, RANK, ROT,
                                                         page, cache.shape[0], 0, 0.07, splits, partial.data_ptr(), None, kernels._stream()), "latent_attention")
    share = partial[0].cpu().double()
    w = torch.exp(share[..., 0] - share[..., 0].amax(1, keepdim=True))
    got = (share[..., 2:] * w[..., None]).sum(1) / (share[..., 1] * w).sum(1)[:, None]
    off = got / expected(q, rows, 0, n, None, 0.07, None, page, ()) - 1
    # an instruction cuts less than 2^-23 of what it holds off, and holds 32 keys' terms at a time; the rest is rounded both ways
    assert off.mean().abs() <= 2.0 ** -23 and off.abs().max() <= 2.0 ** -20, (off.mean(), off.abs().max())
