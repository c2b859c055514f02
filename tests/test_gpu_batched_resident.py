"""Batched solves in one launch over all domains (whole, or the coarse parts)
against each domain stepped alone with a launch per pass: bit for bit, with the
same cycles and decisions.

Sizes: rows that are no multiple of four over a level that stops halving, uneven
mixes, a batch whose coarse parts alone fit the chip, one that does not fit.
"""
import pytest
import torch

from fluxfx_b200.backend.batched import BatchedSmoke, batched_scenes, build_solvers

pytestmark = pytest.mark.gpu

CELL = 1.0 / 64.0


@pytest.mark.parametrize('count,sizes,first', [(1, (32,), 0), (3, (34, 42), 0), (7, (32, 48), 0), (3, (96,), 1),
                                               (4, (128,), -1)])
@pytest.mark.parametrize('warm', [False, True])
def test_batches_match_separate_passes(count, sizes, first, warm):
    from fluxfx_b200.backend.device import CudaDevice
    device, steps = CudaDevice(), 2
    scenes = batched_scenes(count, seed=40 + count, sizes=sizes, warm_start=warm, coarse_scale=1.9 if warm else 1.0)
    alone, sources = build_solvers(scenes, device)
    cycles = []
    for s, src in zip(alone, sources):
        s.projector.use_resident = False
        dt, mine = 0.02, []
        for _ in range(steps):
            s.step(dt, sources=src)
            mine.append(s.projector.last_cycles)
            umax = max(s.projector.velocity_maxima())
            dt = min(0.02, 0.5 * CELL / umax) if umax > 0 else 0.02
        cycles.append(mine)
    solvers, sources = build_solvers(scenes, device)
    batch = BatchedSmoke(solvers, sources)
    assert batch.lib.ffx_batch_resident_first(batch.plan) == first
    batch.run(1)
    batch.run(steps - 1)
    stats = batch.stats()
    for i, s in enumerate(alone):
        density, temperature, velocity = batch.fields(i)
        assert torch.equal(density, s._front) and torch.equal(temperature, s._temperature)
        assert all(torch.equal(a, b) for a, b in zip(velocity, s._velocity))
        assert stats[i]['total_cycles'] == sum(cycles[i]) and stats[i]['last_cycles'] == cycles[i][-1]
    # a decision before every cycle of the domain with the most, and one after them
    assert stats[0]['loop_iterations'] == sum(max(c[k] for c in cycles) + 1 for k in range(steps))
    batch.close()
