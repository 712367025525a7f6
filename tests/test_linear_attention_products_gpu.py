"""Gated linear attention in chunks: what a query reads of every earlier token, one by one.  Queries and keys of ones, decays alike in all channels, no
state and values that tell the tokens apart, so that a result is the product of the decays between two tokens times a power of two: sums of equal
numbers are exact, and what is left is how the decays' product was rounded."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
def test_decays_between_two_tokens(seed):
    from prefixserve_b200 import ops
    from prefixserve_b200.ops import library
    n, dim = 128, 64
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    ctx = types.SimpleNamespace(item_start=dev([0, n]), slots=dev([0]), num_items=1, max_new_tokens=n)
    alpha = 0.3 + 0.7 * torch.rand(n, 1, generator=g, device="cuda")
    proj = torch.cat([torch.ones(n, 2 * dim, device="cuda"), torch.eye(n, device="cuda")], 1).bfloat16()
    before = library.launch_counts.copy()
    out = ops.linear_attention(proj, alpha.repeat(1, dim), torch.zeros(1, dim * n, device="cuda"), ctx, heads=1, dim=dim, vdim=n).double().view(n, n)
    assert (library.launch_counts - before)["linear_attention_chunks"] == 1
    a, want = alpha[:, 0].double(), torch.zeros(n, n, dtype=torch.float64, device="cuda")
    for j in range(n):
        want[j:, j] = dim ** 0.5 * torch.cumprod(torch.cat([torch.ones(1, dtype=torch.float64, device="cuda"), a[j + 1:]]), 0)
    ulps = ((out - want) / want).abs()[torch.tril(torch.ones(n, n, device="cuda")) > 0] * 2.0 ** 24
    i, j = torch.tril_indices(n, n, device="cuda")
    diagonal = i // 16 == j // 16
    # within sixteen tokens a product carries what its roundings lose, and is rounded once; elsewhere it is made of a few such products (tokens to a half's
    # end, chunks, up to the token), each rounded, and sums over 128 channels
    assert float(ulps[diagonal].max()) <= 1.01
    assert float(ulps.max()) <= 24
