"""Gated products whose gate is far below zero: silu(g) is then g e^g, down to the smallest normal numbers, and a large second branch brings it back into
sight.  The sum 1 + e^-g lies between 2^126 and 2^128, where a quick division would answer zero."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0, 256, 512])
@pytest.mark.parametrize("form", ["silu", "scaled", "clipped"])
def test_gates_far_below_zero(form, width):
    from prefixserve_b200.ops import library, tensorcore
    from prefixserve_b200.ops.kernels import _stream
    m, n, k, lib = 256, 128, 64, library.lib()
    alpha = 1.702 if form == "clipped" else 1.0
    gates = torch.tensor([-87.5, -88.0, -87.75, -20.0], device="cuda").repeat(n // 4) / alpha
    x, w = torch.zeros(m, k, device="cuda"), torch.zeros(2 * n, k, device="cuda")
    x[:, 0] = 1
    w[:n, 0], w[n:, 0] = gates, 2.0 ** 100
    x, w = x.bfloat16(), w.bfloat16()
    out, names = torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.zeros(m // 128, dtype=torch.int32, device="cuda")
    scale = torch.ones(m, device="cuda")
    at = (x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, 1, names.data_ptr())
    library.check(lib.psb_gemm_tcgen05_tile_width(width), "tile width")
    try:
        if form == "silu":
            out = tensorcore.gemm_tcgen05_gated(x, w)
        elif form == "scaled":
            library.check(lib.psb_gemm_tcgen05_grouped_gated_silu(*at, scale.data_ptr(), 148, _stream()), "grouped")
        else:
            library.check(lib.psb_gemm_tcgen05_grouped_gated_clipped(*at, 2.0 ** 101, alpha, 0.0, 148, _stream()), "grouped")
    finally:
        library.check(lib.psb_gemm_tcgen05_tile_width(0), "tile width")
    g = w[:n, 0].double()
    want = g / (1 + torch.exp(-alpha * g)) * 2.0 ** 100
    assert float(want.abs().min()) > 1e-8 and math.log2(float((1 + torch.exp(-alpha * g)).max())) < 128
    # __expf multiplies by log2(e) in float32: 88 * 2^-24 of a relative error in the power; the result in bfloat16
    assert ((out.double() - want).abs() <= (2.0 ** -8 + 2e-4) * want.abs()).all()
    assert lib.psb_tcgen05_status() == 0
