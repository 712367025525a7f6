"""Grouping of (token, expert) pairs by expert, one block (fewer than 1,024 pairs) and a cluster of eight, and the copy of the tokens' rows in that order:
every pair one row of its expert's run, runs at multiples of ``pad``, the rest nobody's."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs, experts, pad, top", [(1, 1, 1, 1), (96, 512, 128, 3), (1023, 7, 128, 1), (1024, 7, 128, 4), (1025, 512, 1, 5), (8148, 32, 128, 4),
                                                      (16385, 33, 128, 5), (40000, 8, 64, 8)])
@pytest.mark.parametrize("spread", ["even", "one", "few"])
def test_pairs_by_expert(pairs, experts, pad, top, spread):
    from prefixserve_b200.ops import library
    from prefixserve_b200.ops.kernels import _stream
    lib, g = library.lib(), torch.Generator(device="cuda").manual_seed(pairs)
    i32 = dict(dtype=torch.int32, device="cuda")
    chosen = torch.randint(0, {"even": experts, "one": 1, "few": min(3, experts)}[spread], (pairs,), generator=g, device="cuda", dtype=torch.int32)
    if spread != "even":
        chosen = experts - 1 - chosen
    weight = torch.rand(pairs, generator=g, device="cuda")
    room = -(-(pairs + experts * (pad - 1)) // pad) * pad
    offsets, row_pair, pair_row, tiles = torch.full((experts + 1,), -7, **i32), torch.full((room,), -7, **i32), torch.full((pairs,), -7, **i32), torch.full((room // pad,), -7, **i32)
    row_weight = torch.full((room,), -7.0, device="cuda")
    library.check(lib.psb_moe_group(chosen.data_ptr(), offsets.data_ptr(), row_pair.data_ptr(), pair_row.data_ptr(), tiles.data_ptr(), pairs, experts, pad, room,
                                    weight.data_ptr(), row_weight.data_ptr(), _stream()), "moe_group")
    count = torch.bincount(chosen.long(), minlength=experts)
    start = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), (-(-count // pad) * pad).cumsum(0)])
    assert torch.equal(offsets.long(), start)
    row, e = pair_row.long(), chosen.long()
    assert ((row >= start[e]) & (row < start[e] + count[e])).all() and torch.equal(row_pair[row].long(), torch.arange(pairs, device="cuda"))
    assert torch.equal(row_weight[row], weight)
    nobody = torch.ones(room, dtype=torch.bool, device="cuda")
    nobody[row] = False
    assert (row_pair[nobody] == -1).all() and (row_weight[nobody] == 0).all()
    want = torch.full((room // pad,), -1, dtype=torch.long)
    for i in range(experts):
        want[int(start[i]) // pad: int(start[i + 1]) // pad] = i
    assert torch.equal(tiles.cpu().long(), want)
    for k in (8, 264, 2048, 2120):
        x = torch.randn(-(-pairs // top), k, generator=g, device="cuda").bfloat16()
        rows = torch.full((min(room, 4000), k), 7.0, dtype=torch.bfloat16, device="cuda")
        library.check(lib.psb_moe_gather(x.data_ptr(), row_pair.data_ptr(), rows.data_ptr(), len(rows), k, top, _stream()), "moe_gather")
        of = row_pair[: len(rows)].long()
        assert torch.equal(rows[of >= 0], x[of[of >= 0] // top]) and (rows[of < 0] == 7.0).all()
