"""The barriers of the cluster product's ring (csrc/gemm_cluster.cu) as the library plans them, on the host: a producer that refills
in batches, loads that land out of order, issuers that take the K blocks in turn and wait by parity."""
import random

import pytest

from lia_rs_b200.kernels import ops


def early(stages, bars, issuers, batch, blocks, seed):
    """What an issuer multiplied before it had landed (None: nothing), under one random schedule; a schedule that stops is an error."""
    rng = random.Random(seed)
    completed, freed, in_flight = [0] * bars, [0] * stages, {}              # in flight: block -> time at which it lands
    issued, at, now = min(blocks, stages), list(range(issuers)), 0.0
    ready = [0.0] * issuers
    slow = rng.choice((0.0, 0.05, 0.3))
    landing = lambda: now + rng.uniform(1, 4) * (4 if rng.random() < slow else 1)
    for it in range(issued):
        in_flight[it] = landing()
    while any(it < blocks for it in at):
        now += 0.25
        for it in [it for it, when in in_flight.items() if when <= now]:
            del in_flight[it]
            assert completed[it % bars] == it // bars, "fills of a barrier complete out of turn"
            completed[it % bars] += 1
        nexts = range(issued, min(issued + batch, blocks))
        if nexts and all((freed[it % stages] & 1) != ((it // stages) & 1) ^ 1 for it in nexts):
            for it in nexts:
                assert freed[it % stages] == it // stages, "a stage is filled before it is free"
                in_flight[it] = landing()
            issued = nexts[-1] + 1
        for who in rng.sample(range(issuers), issuers):
            it = at[who]
            if it >= blocks or ready[who] > now or (completed[it % bars] & 1) == ((it // bars) & 1):
                continue
            if it >= issued or it in in_flight:
                return it
            freed[it % stages] += 1
            at[who], ready[who] = it + issuers, now + rng.uniform(0.2, 2.0)
        assert now < 100.0 * blocks + 100.0, "no progress"
    return None


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("n_tile", range(16, 129, 16))
def test_a_barrier_has_one_issuer_and_sees_every_fill(gated, n_tile):
    for blocks in (1, 2, 3, 5, 7, 9, 11, 12, 16, 17, 40):
        stages, bars, issuers, batch = ops.gemm_cluster_ring(gated, n_tile, blocks)
        assert 1 <= batch <= stages <= bars and bars % stages == 0
        for bar in range(bars):
            assert len({it % issuers for it in range(bar, 4 * bars, bars)}) == 1 or blocks <= stages
        for seed in range(60):
            assert early(stages, bars, issuers, batch, blocks, seed) is None, (stages, bars, blocks, seed)


def test_the_model_catches_a_stage_that_two_issuers_share():
    assert any(early(5, 5, 2, 2, 16, seed) is not None for seed in range(400))
