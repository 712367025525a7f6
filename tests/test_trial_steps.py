"""The steps that the engine sizes its pool by hold nearly as many chunks of the recurrences, and so as much of their scratch, as any step that the
scheduler may make of the same budget, requests and longest sequence."""

import pytest

from prefixserve_b200.engine.engine import trial_steps


def most_chunks(budget, requests, longest, least):
    """Over all portions of at least ``least`` tokens: only the shortest that make up so many chunks are worth trying."""
    sizes = [least] + [n for n in range(33, min(budget, longest) + 1, 32) if n > least]
    best = [0] * (budget + 1)
    for _ in range(requests):
        best = [max([best[b]] + [best[b - n] + -(-n // 32) for n in sizes if n <= b and n <= longest]) for b in range(budget + 1)]
    return best[budget]


@pytest.mark.parametrize("budget, requests, longest", [(512, 64, 4096), (512, 8, 4096), (256, 40, 100), (400, 10, 64), (300, 1, 4096), (700, 100, 700), (200, 10, 33),
                                                       (40, 64, 4096), (7, 3, 50), (1, 2, 9)])
def test_chunks_of_the_trial_steps(budget, requests, longest):
    steps = trial_steps(budget, requests, longest)
    for new in steps:
        assert len(new) == requests and max(new) <= longest and min(new) >= 1 and sum(n for n in new if n > 1) <= budget
    assert max(max(new) for new in steps) == min(budget, longest)
    for least in (8, 32):   # from which portions on the delta rules go in chunks, and linear attention
        held = max(sum(-(-n // 32) for n in new if n >= least) for new in steps)
        most = most_chunks(budget, requests, longest, least) if least <= min(budget, longest) else 0
        assert held * 8 >= most * 7, (least, held, most)
