"""Which tcgen05 products go two CTAs a tile of 256 rows (no GPU needed): where both ways were measured, the rule takes the quicker one."""

import pytest

from prefixserve_b200.ops import library


def room(experts, rows):   # of a routed step with so many (token, expert) pairs an expert
    return -(-experts * (rows + 127) // 128) * 128


@pytest.mark.parametrize("experts, rows, n, k, pairs", [
    (32, 8, 2048, 2048, False), (32, 48, 2048, 2048, True), (32, 256, 2048, 2048, True), (32, 8, 2048, 1024, False), (32, 100, 2048, 1024, True),
    (8, 32, 2048, 2048, False), (8, 160, 2048, 1024, False), (64, 8, 1536, 2048, False), (64, 64, 1536, 2048, True), (64, 8, 2048, 768, False),
    (128, 4, 1536, 2048, True), (32, 8, 4096, 4096, True), (32, 64, 4096, 2048, True), (64, 8, 1024, 512, False), (64, 256, 1024, 512, False)])
def test_grouped(experts, rows, n, k, pairs):
    assert bool(library.lib().psb_gemm_tcgen05_pairs(room(experts, rows), n, k, experts, 0, 148)) == pairs


@pytest.mark.parametrize("m, n, k, gated, pairs", [(1979, 4096, 14336, 0, True), (1024, 4096, 14336, 0, True), (700, 4096, 14336, 0, False),
                                                   (1979, 3072, 2048, 0, False), (1024, 14336, 4096, 1, True)])
def test_dense(m, n, k, gated, pairs):
    assert bool(library.lib().psb_gemm_tcgen05_pairs(m, n, k, 0, gated, 148)) == pairs


def test_more_row_tiles_than_a_pair_of_ctas_lists():
    lib = library.lib()
    assert lib.psb_gemm_tcgen05_pairs(128 * 2048, 4096, 4096, 32, 0, 148) == 1
    for width in (0, 512):   # also where a test asks for pairs
        assert lib.psb_gemm_tcgen05_tile_width(width) == 0
        try:
            assert lib.psb_gemm_tcgen05_pairs(128 * 2049, 4096, 4096, 32, 0, 148) == 0
        finally:
            lib.psb_gemm_tcgen05_tile_width(0)
