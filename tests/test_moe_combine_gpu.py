"""The sum over a token's experts (and the shared one) where a block takes two tokens, and around the number of tokens from which it does, against float64.

Bound: a result is a float32 sum of top + 1 products, each step rounded (and the weight of the shared expert, a sigmoid of some 3 units of the last place): (top + 4) 2^-23 of
the sum of the products' sizes; a bfloat16 result rounds once more, 2^-8 of itself."""

import pytest
import torch

from prefixserve_b200.ops import library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top", [1, 4, 5])
@pytest.mark.parametrize("past", [-1, 0, 1])
@pytest.mark.parametrize("shared, out_dtype, h", [(None, torch.bfloat16, 264), (torch.bfloat16, torch.bfloat16, 2056), (torch.bfloat16, torch.float32, 8), (torch.float32, torch.bfloat16, 264)])
def test_two_tokens_a_block(top, past, shared, out_dtype, h):
    tokens = 8 * torch.cuda.get_device_properties(0).multi_processor_count + past  # two tokens a block from 8 a multiprocessor on
    gen = torch.Generator(device="cuda").manual_seed(top + h)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    rows = tokens * top + 200
    y = rand(rows, h).bfloat16()
    pair_row = torch.randperm(rows, generator=gen, device="cuda")[: tokens * top].to(torch.int32)
    weight = torch.rand(tokens, top, generator=gen, device="cuda")
    weight[tokens // 2:] *= 1e-3
    for gated in (False, True) if shared else (False,):
        s = rand(tokens, h).to(shared) if shared else None
        gate = rand(tokens, 3) * 3
        behind = 2
        out = torch.full((tokens + behind, h), 7.0, dtype=out_dtype, device="cuda")
        library.check(library.lib().psb_moe_combine(
            y.data_ptr(), 1, pair_row.data_ptr(), weight.data_ptr(), s.data_ptr() if shared else None, 1 if shared == torch.bfloat16 else 0,
            gate.data_ptr() if gated else None, 3, out.data_ptr(), 1 if out_dtype == torch.bfloat16 else 0, tokens, h, top, library.stream_handle()), "moe_combine")
        terms = [y[pair_row.view(tokens, top)[:, k].long()].double() * weight[:, k: k + 1].double() for k in range(top)]
        if shared:
            terms.append(s.double() * (torch.sigmoid(gate[:, :1].double()) if gated else 1.0))
        want, size = sum(terms), sum(t.abs() for t in terms)
        allowed = (top + 4) * 2.0 ** -23 * size + (2.0 ** -8 * want.abs() if out_dtype == torch.bfloat16 else 0.0)
        assert bool(((out[:tokens].double() - want).abs() <= allowed).all())
        assert bool((out[tokens:] == 7.0).all())
