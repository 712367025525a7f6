"""Single tokens' attention over cache rows fed by the TMA unit against the same in float64: windows, chunks, kept first keys in the
window's own runs and in runs of their own, capped scores, a distance bias, sinks and gates, one to eight heads a key/value head, keys
in one share and in many; pages that nobody has written or that have been given back (NaN, and no number in the table)."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def seen_keys(i, window, chunk, keep):
    j = torch.arange(i + 1)
    seen = torch.ones(i + 1, dtype=torch.bool)
    if window:
        seen &= (i - j < window) | (j < keep)
    if chunk:
        seen &= j // chunk == i // chunk
    return seen


@pytest.mark.parametrize("hq,hkv,page,options", [
    (4, 1, 16, dict(window=200)),
    (8, 1, 16, dict(window=None, sink=True)),
    (3, 3, 16, dict(window=1)),
    (6, 2, 64, dict(window=65, sink=True, gate=True)),
    (4, 2, 16, dict(window=100, softcap=3.0, gate=True, out_scale=-0.5)),
    (4, 1, 32, dict(window=90, keep=4, sink=True)),
    (2, 1, 16, dict(window=64, keep=70)),
    (10, 2, 16, dict(chunk=256, bias=256, sink=True)),
    (2, 1, 16, dict(chunk=100, bias=30)),
])
@pytest.mark.parametrize("least", [1 << 20, 128, 16])
def test_single_tokens(hq, hkv, page, options, least, monkeypatch):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels, library
    monkeypatch.setattr(kernels, "ROWS_DECODE_KEYS_PER_SPLIT", least)   # one share, a few, as many as there may be
    monkeypatch.setattr(kernels, "ROWS_DECODE_BLOCK_SHARE", 1)
    monkeypatch.setattr(kernels, "ROWS_DECODE_LEAST", 0)
    window, chunk, keep = options.get("window"), options.get("chunk"), options.get("keep", 0)
    positions = [0, 15, 16, 63, 99, 255, 256, 700, 1500]
    g = torch.Generator().manual_seed(hq + page + len(options))
    rnd = lambda *s: torch.randn(*s, generator=g)
    t = len(positions)
    need = [p // page + 1 for p in positions]
    ids = torch.randperm(sum(need), generator=g).tolist()
    table = torch.full((t, max(need)), -1, dtype=torch.int32)
    kv = torch.full((sum(need), 1, hkv, page, 2 * D), float("nan"), dtype=torch.bfloat16)
    rows = [rnd(p + 1, hkv, 2 * D).bfloat16() for p in positions]
    for i, p in enumerate(positions):
        seen = seen_keys(p, window, chunk, keep)
        for j in range(need[i]):
            if seen[j * page: (j + 1) * page].any():
                table[i, j] = pid = ids.pop()
                part = rows[i][j * page: (j + 1) * page]
                kv[pid, 0, :, : len(part)] = part.transpose(0, 1)
    q = rnd(t, hq, D).bfloat16()
    sink = 2.0 * rnd(hq) if options.get("sink") else None
    bias = rnd(hq, options["bias"]) if "bias" in options else None
    gate = rnd(t, hq * D + 3).bfloat16() if options.get("gate") else None
    wide = torch.full((t, hq * D + 5), 7.0, dtype=torch.bfloat16, device="cuda")
    dev = lambda x, d=None: None if x is None else torch.as_tensor(x, dtype=d).cuda()
    ctx = types.SimpleNamespace(positions=dev(positions, torch.int32), token_item=dev(list(range(t)), torch.int32),
                                item_start=dev(list(range(t + 1)), torch.int32), num_items=t, max_new_tokens=1, max_kv_len=1501, extras={})
    before = library.launch_counts.copy()
    out = ops.attention_over_rows(q.cuda(), kv.cuda(), table.cuda(), ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=page, scale=0.2,
                                  window=window, chunk=chunk, keep_first=keep, bias=dev(bias), sink=dev(sink), softcap=options.get("softcap"),
                                  gate=None if gate is None else gate.cuda()[:, 3:], out_scale=options.get("out_scale", 1.0), out=wide[:, 5:])
    taken = library.launch_counts - before
    span = min(window + keep if window else 1501, chunk or 1501, 1501)
    assert taken["attention_rows_single"] == 1 and (taken["attention_rows_merge"] == 1) == (span // least >= 2)
    assert bool((wide[:, :5] == 7.0).all())
    got = out.cpu().double().view(t, hq, D)
    for i, p in enumerate(positions):
        keys, values = (x.double().repeat_interleave(hq // hkv, 1) for x in (rows[i][..., :D], rows[i][..., D:]))
        scores = torch.einsum("hd,jhd->hj", q[i].double(), keys) * 0.2
        if options.get("softcap"):
            scores = options["softcap"] * torch.tanh(scores / options["softcap"])
        if bias is not None:
            scores = scores + bias.double()[:, (p - torch.arange(p + 1)).clamp(0, options["bias"] - 1)]
        scores = scores.masked_fill(~seen_keys(p, window, chunk, keep), float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink.double()[:, None]], 1)
        want = torch.einsum("hj,jhd->hd", torch.softmax(scores, 1)[:, : p + 1], values) * options.get("out_scale", 1.0)
        if gate is not None:
            want = want * torch.sigmoid(gate[i, 3:].double().view(hq, D))
        # rounding of the result to bfloat16 (2^-9); weights to 16 bits (2^-17 of values up to 5) and float32 scores up to 100
        assert ((got[i] - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4).all(), (i, p, (got[i] - want).abs().max())
    assert library.tcgen05_status() == 0


@pytest.mark.parametrize("least", [1 << 20, 16])
def test_the_lowest_bias_is_finite(least, monkeypatch):
    """A distance bias of the type's lowest value masks a key beside others; keys that all have it weigh the same."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels
    monkeypatch.setattr(kernels, "ROWS_DECODE_KEYS_PER_SPLIT", least)
    monkeypatch.setattr(kernels, "ROWS_DECODE_BLOCK_SHARE", 1)
    monkeypatch.setattr(kernels, "ROWS_DECODE_LEAST", 0)
    positions, heads = [0, 40, 199], 4
    g = torch.Generator().manual_seed(3)
    kv = torch.randn(3 * 13, 1, 1, 16, 2 * D, generator=g).bfloat16()
    table = torch.arange(3 * 13, dtype=torch.int32).view(3, 13)
    q = torch.randn(3, heads, D, generator=g).bfloat16()
    bias = torch.randn(heads, 300, generator=g)
    bias[1] = bias[2, 50:] = bias[3, :30] = torch.finfo(torch.float32).min
    dev = lambda x: torch.tensor(x, dtype=torch.int32).cuda()
    ctx = types.SimpleNamespace(positions=dev(positions), token_item=dev([0, 1, 2]), item_start=dev([0, 1, 2, 3]), num_items=3, max_new_tokens=1,
                                max_kv_len=200, extras={})
    out = ops.attention_over_rows(q.cuda(), kv.cuda(), table.cuda(), ctx, num_heads=heads, num_kv_heads=1, dim=D, vdim=D, page_size=16, scale=0.1,
                                  bias=bias.cuda()).cpu().double().view(3, heads, D)
    for i, p in enumerate(positions):
        rows = kv[table[i].long()].reshape(-1, 2 * D)[: p + 1].double()
        scores = q[i].double() @ rows[:, :D].t() * 0.1 + bias.double()[:, p - torch.arange(p + 1)]
        want = torch.softmax(scores, 1) @ rows[:, D:]
        # as in test_single_tokens
        assert ((out[i] - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4).all(), (i, p)
