"""Epilogues of the tcgen05 product with two CTAs a tile against one CTA a tile, bit for bit: the projection that rotates and appends to the pages (heads
whose angles stay in registers, and other sizes, whose columns two warps share), the clipped gate, and functions of the sum in rows of a wider tensor."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def at_widths(call, widths=(512, 256)):
    from prefixserve_b200.ops import library
    got = []
    for width in widths:
        library.check(library.lib().psb_gemm_tcgen05_tile_width(width), "tile width")
        try:
            got.append(call())
        finally:
            library.check(library.lib().psb_gemm_tcgen05_tile_width(0), "tile width")
    assert library.lib().psb_tcgen05_status() == 0
    return got


@pytest.mark.parametrize("m", [1, 128, 129, 300, 900])
@pytest.mark.parametrize("hq, hkv, d, k", [(8, 2, 64, 512), (4, 4, 128, 200), (6, 2, 128, 520), (3, 1, 48, 96), (5, 2, 16, 72), (3, 2, 80, 264), (4, 1, 96, 1024)])
def test_rotating_projection(m, hq, hkv, d, k):
    from prefixserve_b200.ops import library
    from prefixserve_b200.ops.kernels import _stream
    page, most = 16, 1200
    g = torch.Generator(device="cuda").manual_seed(m + d + k)
    i32 = lambda x: x.to(torch.int32).cuda()
    requests = 3 if m > 2 else 1
    held = torch.tensor([0, 37, 200][:requests])
    new = torch.tensor([m - m // 3 - m // 5, m // 3, m // 5][:requests]) if requests > 1 else torch.tensor([m])
    positions = i32(torch.cat([torch.arange(o, o + n) for o, n in zip(held, new)]))
    token_item = i32(torch.repeat_interleave(torch.arange(requests), new))
    wide = int(-(-(held + new).max() // page))
    table = i32(torch.randperm(requests * wide, generator=torch.Generator().manual_seed(m)).view(requests, wide))
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn((hq + 2 * hkv) * d, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    angles = torch.outer(torch.arange(most).float(), 1.0 / (10000.0 ** (torch.arange(0, d, 2).float() / d))).cuda()
    cos, sin = angles.cos().contiguous(), angles.sin().contiguous()

    def call():
        kv, q = torch.full((requests * wide, 2, hkv, page, d), 7.0, dtype=torch.bfloat16, device="cuda"), torch.empty(m, hq, d, dtype=torch.bfloat16, device="cuda")
        library.check(library.lib().psb_gemm_tcgen05_rope(x.data_ptr(), w.data_ptr(), m, k, 148, positions.data_ptr(), token_item.data_ptr(), table.data_ptr(), wide,
                                                          cos.data_ptr(), sin.data_ptr(), kv.data_ptr(), q.data_ptr(), hq, hkv, d, page, requests * wide, most,
                                                          _stream()), "rope")
        return q, kv

    (q2, kv2), (q1, kv1) = at_widths(call)
    assert torch.equal(q2, q1) and torch.equal(kv2, kv1)
    untouched = torch.ones(requests * wide, page, dtype=torch.bool)
    for i in range(requests):
        for p in range(int(held[i]), int(held[i] + new[i])):
            untouched[int(table[i, p // page]), p % page] = False
    assert (kv2.transpose(2, 3)[:, :, :][untouched.cuda()[:, None].expand(-1, 2, -1)] == 7.0).all()
    # values are the product's columns as they are: bfloat16 of float32 sums
    want = (x.double() @ w[(hq + hkv) * d:].double().t()).view(m, hkv, d)
    got = kv2[table.long()[token_item.long(), positions.long() // page], 1, :, positions.long() % page].double()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * k ** 0.5).all()


@pytest.mark.parametrize("m, n, k", [(1, 8, 8), (129, 264, 72), (600, 1000, 384)])
def test_clipped_gate_and_functions_of_the_sum(m, n, k):
    from prefixserve_b200.ops import library
    from prefixserve_b200.ops.kernels import _stream
    lib = library.lib()
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, w = (torch.randn(a, k, generator=g, device="cuda").bfloat16() for a in (m, 2 * n))
    expert = torch.zeros(-(-m // 128), dtype=torch.int32, device="cuda")

    def clipped():
        out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        library.check(lib.psb_gemm_tcgen05_gated_clipped(x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, 148, 7.0, 1.702, 1.0, _stream()), "clipped")
        return out

    def unary(kind):
        out = torch.full((m, n + 16), 7.0, dtype=torch.bfloat16, device="cuda")
        library.check(lib.psb_gemm_tcgen05_unary(x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, n + 16, 148, kind, _stream()), "unary")
        assert (out[:, n:] == 7.0).all()
        return out

    def squared():
        out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        library.check(lib.psb_gemm_tcgen05_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, 1, expert.data_ptr(), 1, 148, _stream()), "relu2")
        return out

    for call in (clipped, lambda: unary(0), lambda: unary(1), squared):
        pair, single = at_widths(call)
        assert torch.equal(pair, single)
