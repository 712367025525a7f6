"""What the ops ask of a step's requests when they choose among kernels: from the requests where the host holds them, and safe
bounds where it does not (no list of them, or an empty one)."""

import types

import pytest

from prefixserve_b200.ops import kernels


def context(lengths, items):
    views = [types.SimpleNamespace(start=7 * i, end=7 * i + n) for i, n in enumerate(lengths)]
    ctx = types.SimpleNamespace(num_items=len(lengths), max_new_tokens=max(lengths))
    if items != "absent":
        ctx.items = {"held": views, "none": None, "empty": []}[items]
    return ctx


@pytest.mark.parametrize("items", ["held", "none", "empty", "absent"])
@pytest.mark.parametrize("lengths", [[16], [300, 1], [128, 129, 15], [1, 1, 40], [16, 16]])
def test_portions(lengths, items):
    ctx, t = context(lengths, items), sum(lengths)
    below = any(n < 16 for n in lengths)
    tiles = sum(-(-n // 128) for n in lengths if n >= 16)
    if items == "held":
        assert kernels._has_portions_below(ctx, 16) == below and kernels._portion_tiles(ctx, t, 16, 128) == tiles
    else:   # never too few tiles, and never none below where there are some
        assert kernels._has_portions_below(ctx, 16) >= below and kernels._portion_tiles(ctx, t, 16, 128) >= tiles
