"""Blocks that share out all runs of keys of a step of single tokens evenly: more tokens than a warp has lanes, pieces that begin and end inside a
token's keys, many pieces a block, many blocks a piece, and rings that go round many times."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


@pytest.mark.parametrize("tokens,hq,hkv,longest,options", [
    (1, 8, 1, 9000, dict(sink=True)), (3, 4, 2, 5000, dict(window=3000, keep_first=20)), (33, 8, 2, 2500, dict()), (70, 8, 8, 1500, dict(window=700, sink=True)),
    (64, 4, 4, 3000, dict(chunk=1024)),
])
def test_shared_out(tokens, hq, hkv, longest, options):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    g = torch.Generator(device="cuda").manual_seed(tokens)
    page = 16
    positions = torch.randint(0, longest, (tokens,), generator=g, device="cuda", dtype=torch.int32)
    positions[0] = longest - 1
    width = -(-longest // page)
    kv = torch.randn(tokens * width, 1, hkv, page, 2 * D, generator=g, device="cuda").bfloat16()
    table = torch.randperm(tokens * width, generator=g, device="cuda").int().view(tokens, width)
    q = torch.randn(tokens, hq, D, generator=g, device="cuda").bfloat16()
    more = dict(options)
    if more.pop("sink", False):
        more["sink"] = torch.randn(hq, generator=g, device="cuda")
    at = torch.arange(tokens + 1, dtype=torch.int32, device="cuda")
    ctx = types.SimpleNamespace(positions=positions, token_item=at[:-1], item_start=at, num_items=tokens, max_new_tokens=1, max_kv_len=longest, extras={})
    got = ops.attention_over_rows(q, kv, table, ctx, num_heads=hq, num_kv_heads=hkv, dim=D, vdim=D, page_size=page, scale=0.1, **more).double().view(tokens, hq, D)
    for i, p in enumerate(positions.tolist()):
        rows = kv[table[i].long()][:, 0].transpose(1, 2).reshape(-1, hkv, 2 * D)[: p + 1].double().repeat_interleave(hq // hkv, 1)
        j = torch.arange(p + 1, device="cuda")
        seen = torch.ones_like(j, dtype=torch.bool)
        if "window" in more:
            seen &= (p - j < more["window"]) | (j < more.get("keep_first", 0))
        if "chunk" in more:
            seen &= j // more["chunk"] == p // more["chunk"]
        scores = (torch.einsum("hd,jhd->hj", q[i].double(), rows[..., :D]) * 0.1).masked_fill(~seen, float("-inf"))
        if "sink" in more:
            scores = torch.cat([scores, more["sink"].double()[:, None]], 1)
        want = torch.einsum("hj,jhd->hd", torch.softmax(scores, 1)[:, : p + 1], rows[..., D:])
        # rounding of the result to bfloat16 (2^-9); weights to 16 bits (2^-17 of values up to 5) and float32 scores up to 100
        assert ((got[i] - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4).all(), (i, p)
    assert library.tcgen05_status() == 0
