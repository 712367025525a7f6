"""The hand-over protocol of the prefill attention kernel with heads of 64 (csrc/kernels/attention_tcgen05.cu), run as a
model on the CPU like the protocols in test_attention_pipeline_model.py, whose parts it uses.

With heads of 64 (128 keys a block) each tile has a warp that issues its P V, and S of the event that takes over the
buffer behind it (of either tile), and each row has two softmax threads, whose warps meet once a block.  What differs from
the other protocols: kv_empty takes an arrival per tile (the second tile's warp also arrives for a first tile that does not
see the block), p_ready takes eight, and S of one tile may be issued by the other tile's warp.
"""

import random

import pytest
from test_attention_pipeline_model import KERNEL, SHAPES, Barrier, Kernel, block_ready, producer, wait

NB = 3  # score buffers with heads of 64


class Halves(Kernel):
    def __init__(self, ntiles, n0, nblk, rng):
        super().__init__(ntiles, n0, nblk, NB, False, True, rng)
        self.kv_empty = [Barrier(ntiles) for _ in range(self.stages)]
        self.p_ready = [Barrier(8) for _ in range(2)]
        self.queues = {0: [], 1: []}                       # one issuing warp per tile

    def first_issuer(self, e):
        return 0                                           # the first S, in order, all from one warp


def issuer(k, mine):
    queue, seen = k.queues[mine], [0]
    for e in range(min(k.nb, k.total)):
        if k.first_issuer(e) != mine:
            continue
        yield from block_ready(k, seen, k.block_of(e))
        queue += [("s", e), ("commit", k.s_full[e % k.nb])]
    for i in range(k.blocks_of_tile(mine)):
        e = k.seq_of(mine, i)
        yield from block_ready(k, seen, i)
        ahead = e + k.nb < k.total
        if ahead:
            yield from block_ready(k, seen, k.block_of(e + k.nb))
        yield from wait(k.p_ready[mine], i & 1, i)
        queue += [("pv", e), ("commit", k.o_full[mine])]
        if k.ntiles == 2 and i >= k.n0:
            k.kv_empty[i % k.stages].arrive()
        queue.append(("commit", k.kv_empty[i % k.stages]))
        if ahead:
            queue += [("s", e + k.nb), ("commit", k.s_full[e % k.nb])]
        yield


def softmax_warp(k, t, met, half):
    """``met`` counts, per half, the blocks whose maximum that half has announced."""
    mine = k.blocks_of_tile(t)

    def request(i):
        e = k.seq_of(t, i)
        yield from wait(k.s_full[e % k.nb], (e // k.nb) & 1, e // k.nb)

    if mine > 0:
        yield from request(0)
    for i in range(mine):
        met[half] += 1
        while met[half ^ 1] <= i:
            yield
        if i > 0:
            yield from wait(k.o_full[t], (i - 1) & 1, i - 1)
        for _ in range(k.rng.randrange(3)):
            yield                   # the exponentials
        asked = False
        if i + 1 < mine:
            e = k.seq_of(t, i + 1)
            if k.s_full[e % k.nb].passes((e // k.nb) & 1):
                assert k.s_full[e % k.nb].completed >= e // k.nb + 1
                asked = True
        k.p_ready[t].arrive()
        if i + 1 < mine and not asked:
            yield from request(i + 1)
    met[half] += 1                  # the sums
    while met[half ^ 1] <= mine:
        yield
    if mine > 0:
        yield from wait(k.o_full[t], (mine - 1) & 1, mine - 1)


def state(k, meetings):
    return (tuple((b.completed, b.pending) for group in (k.kv_full, k.kv_empty, k.s_full, k.p_ready, k.o_full) for b in group),
            tuple(map(tuple, meetings)), len(k.queues[0]), len(k.queues[1]))


def run(ntiles, n0, nblk, seed, kernel=Halves):
    rng = random.Random(seed)
    k = kernel(ntiles, n0, nblk, rng)
    agents, meetings = [producer(k)] + [issuer(k, t) for t in range(ntiles)], []
    for t in range(ntiles):
        for _ in range(4):
            meetings.append([0, 0])
            agents += [softmax_warp(k, t, meetings[-1], half) for half in range(2)]
    quiet = 0
    while agents or any(k.queues.values()):
        moved = False
        if rng.random() < 0.4:
            moved = k.tensor_step()
        elif agents:
            a, before = rng.choice(agents), state(k, meetings)
            try:
                next(a)
            except StopIteration:
                agents.remove(a)
                moved = True
            moved = moved or before != state(k, meetings)
        quiet = 0 if moved else quiet + 1
        assert quiet < 5000, f"nothing moves any more: {len(agents)} agents wait ({ntiles=} {n0=} {nblk=})"
    assert len([x for x in k.ran if x[0] == "pv"]) == k.total


@pytest.mark.parametrize("ntiles,n0,nblk", [s for s in SHAPES if s[2] > 0])
def test_every_small_shape_finishes_without_an_early_pass(ntiles, n0, nblk):
    for seed in range(12):
        run(ntiles, n0, nblk, seed)


def test_the_model_notices_a_missing_arrival():
    """A block is given up by one tile only: the model finds the stage overwritten, or a wait that passes early."""
    class Early(Halves):
        def __init__(self, *a):
            super().__init__(*a)
            self.kv_empty = [Barrier(1) for _ in range(self.stages)]

    with pytest.raises(AssertionError):
        for seed in range(20):
            run(2, 7, 9, seed, Early)


def test_the_model_notices_first_scores_out_of_order():
    """Each tile's warp issuing its own first S: S of event 1 may complete, and tile 1 go on to event 3 (the buffer of
    event 0), before S of event 0 has; its wait for event 3 then passes on the phase before."""
    class Apart(Halves):
        def first_issuer(self, e):
            return self.tile_of(e)

    with pytest.raises(AssertionError):
        for seed in range(400):
            run(2, 2, 3, seed, Apart)


def test_the_kernel_has_what_is_modelled():
    text = KERNEL.read_text()
    for line in ("mbar_init(&bars->kv_empty[s], Sh::TWO_ISSUERS || rows_here <= TILE_M ? 1 : 2);",
                 "mbar_init(&bars->p_ready[t], 2 * SOFTMAX_WARPS);",
                 "static constexpr int HALVES = KB == 128 ? 2 : 1, PART = KB / HALVES;",
                 "if (ntiles == 2 && i >= n0) mbar_arrive(&bars->kv_empty[i % STAGES]);"):
        assert line in text, f"the kernel no longer says: {line}"
