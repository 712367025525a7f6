"""Blocks shared out among tokens of different lengths (latent attention on the tensor cores): more tokens than a warp has lanes, any
number of blocks from one a token up to the most, lengths from one key on, two groups of heads."""

import pytest
import torch

from test_latent_attention_mma_gpu import RANK, case, expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,heads,window,shares", [
    (2, 32, 0, 3), (5, 16, 0, 64), (31, 16, 0, 40), (32, 64, 0, 33), (33, 32, 0, 34), (33, 16, 100, 200), (70, 16, 0, 148), (70, 32, 0, 2240),
])
def test_shares_follow_the_lengths(tokens, heads, window, shares):
    from prefixserve_b200.ops import kernels
    g = torch.Generator().manual_seed(tokens)
    lengths = torch.randint(1, 600, (tokens,), generator=g).tolist()
    lengths[0], lengths[-1] = 1, 1100
    page = 16
    q, cache, table, rows, positions, _ = case(lengths, heads, page, tokens)
    dev = [x.cuda() for x in (q, cache, table, positions, torch.arange(tokens, dtype=torch.int32))]
    out = torch.empty(tokens, heads, RANK, dtype=torch.bfloat16, device="cuda")
    partial = torch.full((shares, heads, RANK + 2), float("nan"), device="cuda")
    ptr = [x.data_ptr() for x in dev]
    kernels.check(kernels.lib().psb_latent_attention_mma(*ptr[:3], table.shape[1], ptr[3], ptr[4], None, out.data_ptr(), tokens, heads, RANK, 64, page,
                                                         cache.shape[0], window, 0.07, shares, partial.data_ptr(), None, kernels._stream()), "latent_attention")
    got = out.cpu().double()
    for i, n in enumerate(lengths):
        want = expected(q, rows, i, n, window, 0.07, None, page, ())
        # the result is rounded to bfloat16 (2^-9 of a value); scores, weights and sums are float32
        assert ((got[i] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all(), (i, n)
    for wrong in (tokens - 1, 32 * tokens + 1):
        assert kernels.lib().psb_latent_attention_mma(*ptr[:3], table.shape[1], ptr[3], ptr[4], None, out.data_ptr(), tokens, heads, RANK, 64, page,
                                                      cache.shape[0], window, 0.07, wrong, partial.data_ptr(), None, kernels._stream()) != 0
