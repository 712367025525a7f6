"""The tcgen05 product with two CTAs on a tile of 256 rows, against the kernel with one CTA a tile of 128: the same sums in the same order, so the
same bits.  Rows and columns at and around the tiles' edges, contractions shorter than the ring and no multiple of its step; grouped products
whose experts have even and odd numbers of row tiles, none, and only one."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def both(call):
    from prefixserve_b200.ops import library
    got = []
    for width in (512, 256):
        library.check(library.lib().psb_gemm_tcgen05_tile_width(width), "tile width")
        try:
            got.append(call())
        finally:
            library.check(library.lib().psb_gemm_tcgen05_tile_width(0), "tile width")
    assert library.lib().psb_tcgen05_status() == 0
    return got


@pytest.mark.parametrize("m, n, k", [(1, 8, 8), (128, 256, 64), (129, 264, 72), (255, 2048, 448), (257, 248, 1000), (600, 1000, 384), (2500, 5000, 512)])
def test_plain_and_gated(m, n, k):
    from prefixserve_b200.ops import tensorcore
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x, w = (torch.randn(a, k, generator=g, device="cuda").bfloat16() for a in (m, n))
    for call in (lambda: tensorcore.gemm_tcgen05(x, w), lambda: tensorcore.gemm_tcgen05_gated(x, w), lambda: tensorcore.gemm_tcgen05_gated(x, w, 1)):
        pair, single = both(call)
        assert torch.equal(pair, single)
    want = x.double() @ w.double().t()
    assert (both(lambda: tensorcore.gemm_tcgen05(x, w))[0].double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("counts, n, k", [([1], 64, 128), ([256, 0, 128, 300, 5], 200, 192), ([0, 0, 700, 129, 0, 384], 520, 64), ([40] * 70, 264, 136)])
@pytest.mark.parametrize("gated", [False, True])
def test_grouped(counts, n, k, gated):
    from prefixserve_b200.ops import library
    from prefixserve_b200.ops.kernels import _stream
    g = torch.Generator(device="cuda").manual_seed(n)
    tiles = [e for e, c in enumerate(counts) for _ in range(-(-c // 128))] + [-1, -1, -1]
    rows, experts = 128 * len(tiles), len(counts)
    x = torch.randn(rows, k, generator=g, device="cuda").bfloat16()
    w = torch.randn(experts, 2 * n if gated else n, k, generator=g, device="cuda").bfloat16()
    scale, names = torch.rand(rows, generator=g, device="cuda"), torch.tensor(tiles, dtype=torch.int32, device="cuda")
    lib = library.lib()

    def call():
        out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
        at = (x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, n, k, experts, names.data_ptr())
        if gated:
            library.check(lib.psb_gemm_tcgen05_grouped_gated_silu(*at, scale.data_ptr(), 148, _stream()), "grouped")
        else:
            library.check(lib.psb_gemm_tcgen05_grouped(*at, 0, 148, _stream()), "grouped")
        return out

    pair, single = both(call)
    assert torch.equal(pair, single)
    assert (pair[128 * (len(tiles) - 3):] == 7.0).all()   # rows of nobody stay as they were
    for t, e in enumerate(tiles[:-3]):
        run = slice(128 * t, 128 * t + 128)
        y = x[run].double() @ w[e].double().t()
        if gated:
            y = y.bfloat16().double()
            r = scale[run, None].double()
            y = torch.nn.functional.silu(r * y[:, :n]) * (r * y[:, n:])
        # a sum that rounds to its neighbour moves gate and up by 2^-8 of themselves
        assert ((pair[run].double() - y).abs() <= 2.0 ** -6 * y.abs() + 2.0 ** -7 * y.abs().max()).all(), t
