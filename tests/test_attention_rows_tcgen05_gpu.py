"""Prompt portions' attention over cache rows on tcgen05 against the same in float64: every mask, a cap on scores near and far
from it, a distance bias with a short reach, kept first keys that lie in the window's own blocks, in blocks of their own and
across several, sinks and gates; portions at the edges of tiles of 128 tokens and of blocks of 64 keys, whole and cut into
ranges of keys; pages that nobody has written or that have been given back (NaN, and no number in the table)."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def step(lengths, starts):
    positions, item_of, offsets = [], [], [0]
    for i, (n, s) in enumerate(zip(lengths, starts)):
        positions += range(s, s + n)
        item_of += [i] * n
        offsets.append(offsets[-1] + n)
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    return types.SimpleNamespace(positions=dev(positions), token_item=dev(item_of), item_start=dev(offsets), num_items=len(lengths),
                                 max_new_tokens=max(lengths), max_kv_len=max(n + s for n, s in zip(lengths, starts)), extras={})


def seen_keys(i, keys, window, chunk, keep):
    j = torch.arange(keys)
    seen = j <= i
    if window:
        seen &= (i - j < window) | (j < keep)
    if chunk:
        seen &= j // chunk == i // chunk
    return seen


@pytest.mark.parametrize("hq,hkv,page,options", [
    (4, 1, 16, dict(window=200)),
    (4, 2, 16, dict(window=None)),
    (3, 1, 8, dict(window=1)),
    (2, 2, 64, dict(window=65, sink=True, gate=True)),
    (4, 2, 16, dict(window=100, softcap=3.0, gate=True)),
    (4, 2, 32, dict(window=300, softcap=500.0, gate=True, out_scale=-0.5)),
    (4, 1, 16, dict(window=90, keep=4, sink=True)),
    (2, 1, 16, dict(window=64, keep=70)),
    (2, 1, 8, dict(window=200, keep=130, sink=True)),
    (4, 2, 16, dict(chunk=256, bias=256, sink=True)),
    (2, 1, 16, dict(chunk=100, bias=30)),
    (2, 1, 16, dict(window=5000, bias=4600)),
])
@pytest.mark.parametrize("ranges", [1, 8])
def test_portions(hq, hkv, page, options, ranges, monkeypatch):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels, library
    monkeypatch.setattr(kernels, "ROWS_TCGEN05_RANGES", ranges)   # every unit a CTA's, or cut into ranges of keys where that pays
    window, chunk, keep = options.get("window"), options.get("chunk"), options.get("keep", 0)
    far = options.get("bias", 0) > 4096   # distances beyond those whose bias the kernel keeps at hand
    lengths, starts = ([200], [4500]) if far else ([64, 300, 1, 129, 20, 256], [0, 331, 500, 1000, 7, 60])
    g = torch.Generator().manual_seed(hq + page + len(options))
    rnd = lambda *s: torch.randn(*s, generator=g)
    ctx, t = step(lengths, starts), sum(lengths)
    held = [n + s for n, s in zip(lengths, starts)]
    need = [-(-n // page) for n in held]
    ids = torch.randperm(sum(need), generator=g).tolist()
    table = torch.full((len(held), max(need)), -1, dtype=torch.int32)
    kv = torch.full((sum(need), 1, hkv, page, 2 * D), float("nan"), dtype=torch.bfloat16)
    rows = [rnd(n, hkv, 2 * D).bfloat16() for n in held]
    for i, n in enumerate(held):
        # what the portion's first token can see and everything behind it; other pages have been given back
        first = seen_keys(starts[i], n, window, chunk, keep)
        first[starts[i]:] = True
        for j in range(need[i]):
            if first[j * page: (j + 1) * page].any():
                table[i, j] = pid = ids.pop()
                part = rows[i][j * page: (j + 1) * page]
                kv[pid, 0, :, : len(part)] = part.transpose(0, 1)
    q = rnd(t, hq, D).bfloat16()
    sink = 2.0 * rnd(hq) if options.get("sink") else None
    bias = rnd(hq, options["bias"]) if "bias" in options else None
    gate = rnd(t, hq * D + 16).bfloat16() if options.get("gate") else None
    wide = torch.full((t, hq * D + 24), 7.0, dtype=torch.bfloat16, device="cuda")
    dev = lambda x: None if x is None else x.cuda()
    before = library.launch_counts.copy()
    out = ops.attention_over_rows(q.cuda(), kv.cuda(), table.cuda(), ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=page, scale=0.2,
                                  window=window, chunk=chunk, keep_first=keep, bias=dev(bias), sink=dev(sink), softcap=options.get("softcap"),
                                  gate=None if gate is None else gate.cuda()[:, 8: 8 + hq * D], out_scale=options.get("out_scale", 1.0),
                                  out=wide[:, 8: 8 + hq * D])
    taken = library.launch_counts - before
    assert taken["attention_rows_tcgen05"] == 1 and taken["attention_biased_mma"] == (0 if far else 1)
    assert bool((wide[:, :8] == 7.0).all()) and bool((wide[:, 8 + hq * D:] == 7.0).all())
    got, at = out.cpu().double().view(t, hq, D), 0
    for i, (n, s) in enumerate(zip(lengths, starts)):
        keys, values = (x.cuda().double().repeat_interleave(hq // hkv, 1) for x in (rows[i][..., :D], rows[i][..., D:]))
        scores = torch.einsum("thd,jhd->thj", q[at: at + n].cuda().double(), keys) * 0.2
        if options.get("softcap"):
            scores = options["softcap"] * torch.tanh(scores / options["softcap"])
        if bias is not None:
            dist = (torch.arange(s, s + n)[:, None] - torch.arange(held[i])[None]).clamp(0, options["bias"] - 1)
            scores = scores + bias.cuda().double()[:, dist.cuda()].transpose(0, 1)
        mask = torch.stack([seen_keys(s + r, held[i], window, chunk, keep) for r in range(n)]).cuda()
        scores = scores.masked_fill(~mask[:, None], float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink.cuda().double()[None, :, None].expand(n, hq, 1)], -1)
        want = torch.einsum("thj,jhd->thd", torch.softmax(scores, -1)[..., : held[i]], values).cpu() * options.get("out_scale", 1.0)
        if gate is not None:
            want = want * torch.sigmoid(gate[at: at + n, 8: 8 + hq * D].double().view(n, hq, D))
        # rounding of the result to bfloat16 (2^-9); weights to 16 bits (2^-17 of values up to 5) and float32 scores up to 100
        assert ((got[at: at + n] - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4).all(), (i, n, s, (got[at: at + n] - want).abs().max())
        at += n
    assert library.tcgen05_status() == 0


def own_rows(lengths, starts, hq, hkv, seed=5):
    """A step of portions with their queries and, in consecutive pages, keys and values."""
    g = torch.Generator().manual_seed(seed)
    held = [n + s for n, s in zip(lengths, starts)]
    width = -(-max(held) // 16)
    table = torch.arange(len(held) * width, dtype=torch.int32).view(len(held), width)
    q = torch.randn(sum(lengths), hq, D, generator=g).bfloat16()
    kv = torch.randn(len(held) * width, 1, hkv, 16, 2 * D, generator=g).bfloat16()
    return step(lengths, starts), q.cuda(), kv.cuda(), table.cuda()


def exact_rows(q, kv, table, lengths, starts, hq, hkv, scale, softcap=None):
    out, at = [], 0
    for i, (n, s) in enumerate(zip(lengths, starts)):
        rows = kv[table[i].long()][:, 0].transpose(1, 2).reshape(-1, hkv, 2 * D)[: n + s].double().repeat_interleave(hq // hkv, 1)
        scores = torch.einsum("thd,jhd->thj", q[at: at + n].double(), rows[..., :D]) * scale
        if softcap:
            scores = softcap * torch.tanh(scores / softcap)
        seen = torch.arange(n + s, device="cuda")[None] <= torch.arange(s, s + n, device="cuda")[:, None]
        out.append(torch.einsum("thj,jhd->thd", torch.softmax(scores.masked_fill(~seen[:, None], float("-inf")), -1), rows[..., D:]).flatten(1))
        at += n
    return torch.cat(out)


@pytest.mark.parametrize("scale", [0.0, -0.1])
@pytest.mark.parametrize("softcap", [None, 3.0])
def test_scales_that_are_not_positive(scale, softcap):
    """They turn the order of the scores around (or make them equal): such calls stay with the kernel on mma.sync."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    lengths, starts = [150, 20], [30, 0]
    ctx, q, kv, table = own_rows(lengths, starts, 4, 2)
    before = library.launch_counts.copy()
    out = ops.attention_over_rows(q, kv, table, ctx, num_heads=4, num_kv_heads=2, dim=D, vdim=D, page_size=16, scale=scale, softcap=softcap)
    assert (library.launch_counts - before)["attention_rows_tcgen05"] == 0
    want = exact_rows(q, kv, table, lengths, starts, 4, 2, scale, softcap)
    # as in test_portions
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4).all()


def test_capped_scores_do_not_depend_on_what_does_not_count():
    """The form of the cap is chosen by the scores of a run of rows: small ones here.  What lies behind a sequence's end in its last
    page, the keys of later tokens, keys in front of the window and the request that follows must not change a bit."""
    from prefixserve_b200 import ops
    lengths, starts, hq, hkv, window = [100, 40], [120, 3], 4, 2, 90
    ctx, q, kv, table = own_rows(lengths, starts, hq, hkv)
    q[:100] *= 0.05
    before = torch.arange(220, device="cuda") < 120 + 1 - window   # out of the first token's window, in a block it reads

    def first_portion(garbage):
        mine, queries = kv.clone(), q.clone()
        queries[100:] = garbage * queries[100:]
        rows = mine[table[0].long()]                   # [pages, 1, hkv, 16, 2 D]
        flat = rows.transpose(1, 3).reshape(-1, hkv, 2 * D)
        flat[220:] = garbage
        flat[:220][before] *= garbage
        mine[table[0].long()] = flat.view(-1, 16, hkv, 1, 2 * D).transpose(1, 3)
        out = ops.attention_over_rows(queries, mine, table, ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=16, scale=0.1,
                                      softcap=20.0, window=window)
        return out[:100]

    assert torch.equal(first_portion(1.0), first_portion(400.0))


@pytest.mark.parametrize("ranges", [1, 8])
def test_gates_far_out(ranges, monkeypatch):
    """Gates between -87.4 and -88.7, where 1 + exp(-gate) lies beyond 2^126, make a value of 2^100 one of about 10^-8, not 0."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels
    monkeypatch.setattr(kernels, "ROWS_TCGEN05_RANGES", ranges)
    lengths, starts, hq, hkv = [60], [400], 2, 1
    ctx, q, kv, table = own_rows(lengths, starts, hq, hkv)
    kv[..., D:] = 2.0 ** 100
    gate = torch.linspace(-88.7, -87.4, 60, device="cuda")[:, None].expand(60, hq * D).contiguous().bfloat16()
    out = ops.attention_over_rows(q, kv, table, ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=16, scale=0.1, gate=gate)
    want = 2.0 ** 100 * torch.sigmoid(gate.double())
    # the result in bfloat16; a factor below the smallest normal number (2^-126) keeps at least 20 bits
    assert (gate.double() > -88.8).all() and ((out.double() / want - 1).abs() <= 2.0 ** -8 + 2.0 ** -16).all()


def views(lengths, starts):
    """The requests of a step as the engine's contexts hold them."""
    return [types.SimpleNamespace(start=s, end=s + n) for n, s in zip(lengths, starts)]


@pytest.mark.parametrize("lengths, starts, softcap", [([1500, 1200], [0, 40], 30.0), ([300, 2000, 16], [700, 0, 90], None)])
def test_more_units_than_the_gpu_holds(lengths, starts, softcap, monkeypatch):
    """Whole units and units cut into ranges of keys in one launch, tiles counted from the requests, nothing left to the kernel on mma.sync."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels, library
    seen, ranges = [], kernels._rows_ranges
    monkeypatch.setattr(kernels, "_rows_ranges", lambda units, *a: seen.append((units,) + ranges(units, *a)) or seen[-1][1:])
    hq, hkv = 16, 4
    ctx, q, kv, table = own_rows(lengths, starts, hq, hkv)
    ctx.items = views(lengths, starts)
    before = library.launch_counts.copy()
    out = ops.attention_over_rows(q, kv, table, ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=16, scale=0.1, softcap=softcap)
    taken = library.launch_counts - before
    assert taken["attention_rows_tcgen05"] == 1 and taken["attention_biased_mma"] == 0
    (units, whole, cut), = seen
    assert units == 8 * sum(-(-n // 128) for n in lengths) and 0 < whole < units and cut > 1
    want = exact_rows(q, kv, table, lengths, starts, hq, hkv, 0.1, softcap)
    # as in test_portions
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4).all()
    assert library.tcgen05_status() == 0


@pytest.mark.parametrize("lengths, runs", [([64, 1, 300, 7, 1], 2), ([1, 1, 15, 16], 1), ([1, 20, 1, 20, 1], 3), ([1, 20, 1, 20, 1, 20, 2], 0)])
@pytest.mark.parametrize("options", [dict(), dict(window=200, softcap=3.0, gate=True, out_scale=-0.5), dict(window=90, keep_first=70, sink=True),
                                     dict(chunk=256, bias=256, sink=True)])
@pytest.mark.parametrize("least", [0, 1 << 30])
def test_single_tokens_and_short_portions_beside_others(lengths, runs, options, least, monkeypatch):
    """They go through the kernels of a decode step, a launch for each of up to three runs of neighbours; by themselves, where the host
    does not hold the requests or there are more runs, through the kernel on mma.sync."""
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import kernels, library
    monkeypatch.setattr(kernels, "ROWS_DECODE_LEAST", least)   # the kernel fed by the TMA unit, and the other one
    starts = [(331 * i + 40) % 700 for i in range(len(lengths))]
    hq, hkv, t = 4, 2, sum(lengths)
    ctx, q, kv, table = own_rows(lengths, starts, hq, hkv)
    g = torch.Generator(device="cuda").manual_seed(1)
    more = {k: v for k, v in options.items() if k not in ("gate", "sink", "bias")}
    if "gate" in options:
        more["gate"] = torch.randn(t, hq * D + 16, generator=g, device="cuda").bfloat16()[:, 8: 8 + hq * D]
    if "sink" in options:
        more["sink"] = torch.randn(hq, generator=g, device="cuda")
    if "bias" in options:
        more["bias"] = torch.randn(hq, options["bias"], generator=g, device="cuda")

    def run():
        before = library.launch_counts.copy()
        wide = torch.full((t, hq * D + 16), 7.0, dtype=torch.bfloat16, device="cuda")
        out = ops.attention_over_rows(q, kv, table, ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=16, scale=0.1, out=wide[:, 8: 8 + hq * D], **more)
        assert bool((wide[:, :8] == 7.0).all()) and bool((wide[:, 8 + hq * D:] == 7.0).all())
        return out.double(), library.launch_counts - before

    want, taken = run()
    assert taken["attention_biased_mma"] == 1 and taken["attention_rows_single"] == 0
    ctx.items = views(lengths, starts)
    got, taken = run()
    assert taken["attention_rows_tcgen05"] == 1 and taken["attention_rows_single"] == runs and taken["attention_biased_mma"] == (runs == 0)
    # two results within test_portions' bound of the exact one
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 6e-4).all()
    assert library.tcgen05_status() == 0
