"""The geometric multigrid projector's own methods and attributes beside its whole
cycles: single V-cycles, and sweep counts set on the projector.

Whole cycles against single ones: both round a cell's update some eight times a
sweep, so after n sweeps they differ by at most 2 x 8 (n + 16) 2^-24 max|p|.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(storage='FP32', shape=(32, 48, 40), **settings):
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.multigrid import MultigridPressureProjector
    from fluxfx_b200.physics.config import GridSpec
    from fluxfx_b200.physics.pressure import PressureSettings
    grid = GridSpec(shape, tuple(n / max(shape) for n in shape))
    projector = MultigridPressureProjector(grid, PressureSettings(storage=storage, **settings), CudaDevice())
    projector.reset()
    g = torch.Generator(device='cuda').manual_seed(2)
    projector.before.copy_(torch.randn(projector.before.shape, generator=g, device='cuda'))
    projector.before.sub_(projector.before.mean())
    return projector


def solve(projector, cycles):
    projector.levels[0]['p'], projector.levels[0]['q'] = projector.pressure, projector.spare
    projector.last_iterations = projector.last_coarse_solves = projector.last_cycles = 0
    projector._cycles(cycles, 1.0, True)
    return projector.levels[0]['p'].clone(), projector.last_iterations, projector.last_coarse_solves


@pytest.mark.parametrize('storage', ['FP32', 'BF16'])
@pytest.mark.parametrize('coarse', ['DIRECT', 'SMOOTH'])
def test_single_cycles(storage, coarse):
    projector = make(storage, (64, 64, 64), coarse_solver=coarse)
    want, iterations, direct = solve(projector, 2)
    assert direct == (2 if coarse == 'DIRECT' else 0)
    projector.levels[0]['p'], projector.levels[0]['q'] = projector.pressure, projector.spare
    projector.pressure.zero_()
    projector.last_iterations = projector.last_coarse_solves = 0
    for _ in range(2):
        projector.cycle(0, 1.0)
    got = projector.levels[0]['p']
    assert (projector.last_iterations, projector.last_coarse_solves) == (iterations, direct)
    bound = 2 * 8 * (iterations + 16) * 2.0 ** -24 * float(want.abs().max())
    assert float((got - want).abs().max()) <= bound
    projector.reset()
    projector.close()


@pytest.mark.parametrize('sweeps', [(1, 2), (5, 3), (0, 4), (2, 0)])
def test_sweep_counts_set_on_the_projector(sweeps):
    """They hold from the next solve on, none on a side included."""
    pre, post = sweeps
    projector = make()
    solve(projector, 1)
    projector.pre_sweeps, projector.post_sweeps = pre, post
    got, iterations, _ = solve(projector, 2)
    levels = len(projector.levels)
    assert iterations == 2 * ((levels - 1) * (pre + post) + 80)
    if pre and post:
        want, _, _ = solve(make(mg_pre_sweeps=pre, mg_post_sweeps=post), 2)
        assert torch.equal(got, want)
    else:
        assert bool(torch.isfinite(got).all()) and float(got.abs().max()) > 0
    projector.close()

@pytest.mark.parametrize('sweeps', [(0, 4), (3, 0)])
def test_sweep_counts_set_on_a_collider_projector(sweeps):
    from tests.test_gpu_graph_resident import build
    results = []
    for resident in (True, False):
        projector, faces = build((32, 32, 32))
        projector.use_resident = resident
        projector.pre_sweeps, projector.post_sweeps = sweeps
        projector.coarse_pre, projector.coarse_post = sweeps
        out = [torch.zeros_like(f) for f in faces]
        projector.project(faces, out, 0.02)
        results.append(projector.pressure.clone())
        projector.close()
    assert torch.equal(*results) and bool(results[0].any())


def test_the_coarse_basis_is_made_for_whole_cycles_only():
    assert make('FP32', (64, 64, 64)).coarse_basis is not None
    projector = make('BF16', (64, 64, 64))
    assert projector.coarse_basis is None and projector.coarse_matrix is not None
    assert solve(projector, 1)[2] == 1
