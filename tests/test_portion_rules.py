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


@pytest.mark.parametrize("lengths, alone", [([2000], False), ([8, 9], False), ([8, 6, 5], True), ([15, 1], True), ([24, 1], False), ([24] + [1] * 32, True),
                                            ([32] + [1] * 200, False), ([30, 25, 6], True), ([40, 7], False), ([1, 1], True)])
def test_delta_steps_that_go_token_by_token(lengths, alone):
    assert kernels._delta_one_by_one(lengths) == alone and not kernels._delta_one_by_one(None)


@pytest.mark.parametrize("lengths, alone", [([128], False), ([100] + [1] * 16, False), ([100] + [1] * 17, False), ([100] + [1] * 64, True), ([129] + [1] * 200, False), ([96] + [32] * 20, False),
                                            ([96, 8], False), ([96, 9], False), ([96] + [31] * 12, True), ([64] + [1] * 8, False), ([64] + [1] * 32, True),
                                            ([48, 16], True), ([129, 31], False)])
def test_linear_attention_steps_that_go_token_by_token(lengths, alone):
    """16 heads; us in chunks and token by token: [100] + [1] * 17 38 and 55, [96, 9] 32 and 47 (both were left token by token by chunks of 64 tokens, which
    were slower there)."""
    assert kernels._linear_one_by_one(lengths) == alone and not kernels._linear_one_by_one(None)


def test_linear_attention_steps_of_fewer_heads():
    assert kernels._linear_one_by_one([100] + [1] * 64, 16) and not kernels._linear_one_by_one([100] + [1] * 64, 8)


def test_portions_counted():
    assert kernels._portions_from(context([8, 7, 33], "held"), 8) == 2 and kernels._portions_from(context([8, 7, 33], "empty"), 8) == 3


@pytest.mark.parametrize("sms, short, apart", [(148, 11, False), (148, 12, True), (132, 10, False), (132, 11, True), (16, 1, False), (16, 2, True)])
def test_short_portions_beside_chunks_of_the_channel_rule(sms, short, apart):
    """By the SMs of the device that runs them (64 blocks a portion)."""
    assert kernels._channel_delta_apart(context([64] + [1] * short, "held"), 64, sms) == apart
    assert kernels._channel_delta_apart(context([64] + [1] * short, "none"), 64, sms) == apart
