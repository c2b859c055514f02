"""Tuning a batch times the passes that its steps launch and no others."""
import pytest

from fluxfx_b200 import _native as N
from fluxfx_b200.backend.batched import TUNABLE, BatchedSmoke, batched_scenes, build_solvers

pytestmark = pytest.mark.gpu


class Recording:
    """The library with the kinds of its tuning launches noted."""

    def __init__(self, lib):
        self.lib, self.kinds = lib, set()

    def __getattr__(self, name):
        entry = getattr(self.lib, name)
        if name != 'ffx_batch_tune_pass':
            return entry

        def noted(plan, kind, stream):
            self.kinds.add(kind)
            return entry(plan, kind, stream)
        return noted


@pytest.mark.parametrize('count,sizes,first', [(2, (32, 48), 0), (3, (96,), 1), (4, (128,), -1)])
def test_passes_of_a_resident_solve_are_not_timed(count, sizes, first, tmp_path):
    from fluxfx_b200.backend.device import CudaDevice
    solvers, sources = build_solvers(batched_scenes(count, seed=5, sizes=sizes), CudaDevice())
    batch = BatchedSmoke(solvers, sources)
    assert batch.lib.ffx_batch_resident_first(batch.plan) == first
    batch.lib = Recording(batch.lib)
    cache = str(tmp_path / 'tuning.json')
    best = batch.tune(repeats=1, cache=cache)
    launched = {k for k in TUNABLE if best[N.PASS_NAMES[k]][2] > 0}
    assert launched == batch.lib.kinds
    solves = set(N.FIXED_TILE_PASSES) | {N.PASS_RESIDUAL_MAX, N.PASS_SMOOTH, N.PASS_RESIDUAL_RESTRICT, N.PASS_PROLONG_SMOOTH}
    assert {N.PASS_VELOCITY, N.PASS_GRADIENT, N.PASS_SCALAR_FINAL} <= launched
    assert bool(launched & solves) == (first != 0)
    assert all(best[N.PASS_NAMES[k]] == (0, 0, 0.0) for k in set(TUNABLE) - launched)
    assert batch.tune(cache=cache) == best
    batch.run(1)
    assert all(s['steps'] == 1 for s in batch.stats())
    batch.close()
