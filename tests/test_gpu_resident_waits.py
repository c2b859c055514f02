"""Waits of resident solves that give up.

Blocks of a launch number their exchanges; a block whose stored number is altered
waits for words that never come, gives up after the bounded wait and runs to its
end, and so do its neighbours.
"""
import ctypes as C

import pytest

from fluxfx_b200 import _native as N

pytestmark = pytest.mark.gpu


def build(**settings):
    from tests.test_gpu_graph_resident import build as make
    return make((32, 32, 32), **settings)


def solve(projector, rhs):
    """A whole solve of ``rhs`` from zero through the projector's plan."""
    import torch
    from fluxfx_b200.backend.device import ptr
    plan = projector._resident(0)[0]
    p = torch.full_like(rhs, 7.0)
    tolerance = projector.settings.pressure_tolerance
    N.check(projector.device.lib.ffx_graph_solve(
        C.byref(plan), ptr(p), ptr(rhs), 0 if tolerance > 0 else 3, 1, tolerance, 9, ptr(projector._counters),
        projector.device.s))
    torch.cuda.synchronize()
    return p


def numbers(projector, entry=None):
    """The plan's stored numbers (exchanges and decisions of every block): the words
    that its record at the workspace's start points to."""
    import torch
    _, workspace = entry or projector._resident(0)
    base = workspace.data_ptr()
    offsets = {v - base for v in workspace[:8192].view(torch.int64).tolist()}
    at = min(o for o in offsets if 0 < o < 8192 and o % 256 == 0)
    return workspace[at:].view(torch.int32)


@pytest.mark.parametrize('settings', [dict(pressure_tolerance=1e-4), dict()])
def test_the_next_solve_of_a_collider_plan_is_right(settings):
    """Blocks that parted ways in a launch (other maxima, other cycle counts) number
    the next one alike."""
    import torch
    projector, _ = build(**settings)
    plan = projector._resident(0)[0]
    assert plan.blocks > 4
    g = torch.Generator(device='cuda').manual_seed(5)
    rhs = torch.randn(projector.before.shape, generator=g, device='cuda')
    rhs[projector.device.mask.bool()] = 0.0
    rhs[:plan.tile[1], :plan.tile[0]] = 0.0       # block 0's tile: alone it sees a zero right-hand side
    want = solve(projector, rhs)
    assert projector.resident_timeouts() == 0
    stored = numbers(projector)
    assert int(stored[0]) == int(stored[2]) > 0   # blocks 0 and 1
    stored[0] += 1000                             # block 0 counts from another number
    solve(projector, rhs)
    assert projector.resident_timeouts() > 0
    stored[0] -= 1000
    before = projector.resident_timeouts()
    for _ in range(2):
        assert torch.equal(solve(projector, rhs), want)
    assert projector.resident_timeouts() == before
    with pytest.raises(N.FfxError):
        projector.check_waits()                   # said once
    projector.close()


def timed_out(error):
    return error.value.status == N.FFX_ERR_TIMEOUT


@pytest.mark.parametrize('settings,shape', [
    (dict(pressure_tolerance=1e-3), (32, 32, 32)), (dict(), (32, 32, 32)),
    (dict(pressure_method='PCG', solid_warm_start=True, pressure_tolerance=1e-3, pressure_max_cycles=3), (160, 160, 112))])
def test_a_collider_step_reports_waits_that_gave_up(settings, shape):
    """At the next readback, or at the latest by the next step; the step after is right."""
    import torch
    from tests.test_gpu_graph_resident import build as make
    projector, faces = make(shape, **settings)
    first = 0 if settings.get('pressure_method') is None else projector._coarse_resident()
    out = [torch.zeros_like(f) for f in faces]

    def project():
        projector.reset()
        projector.project(faces, out, 0.02)
        return projector.pressure.clone()

    want = project()
    assert projector.metrics()['v_cycles'] > 0 and max(projector.velocity_maxima()) > 0
    entry = projector._residents[first]
    for look in (projector.metrics, projector.velocity_maxima, projector.total_cycles, project):
        numbers(projector, entry)[0] += 1000
        projector.project(faces, out, 0.02)
        torch.cuda.synchronize()
        with pytest.raises(N.FfxError) as error:
            look()
        assert timed_out(error)
        assert torch.equal(project(), want)       # the workspace is as new
        assert projector.resident_timeouts() == 0
    projector.close()


@pytest.mark.parametrize('solver', ['JACOBI', 'MULTIGRID'])
def test_a_step_without_colliders_reports_waits_that_gave_up(solver):
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.multigrid import MultigridPressureProjector
    from fluxfx_b200.backend.pressure import PressureProjector
    from fluxfx_b200.physics.config import GridSpec
    from fluxfx_b200.physics.pressure import PressureSettings
    grid = GridSpec((48, 40, 56))
    make = PressureProjector if solver == 'JACOBI' else MultigridPressureProjector
    projector = make(grid, PressureSettings(pressure_iterations=4, pressure_cycles=1), CudaDevice())
    g = torch.Generator(device='cuda').manual_seed(6)
    faces = [torch.rand(s[::-1], generator=g, device='cuda') - 0.5 for s in grid.face_shapes]
    out = [torch.zeros_like(f) for f in faces]

    def project():
        projector.reset()
        projector.project(faces, out, 0.02)
        return projector.pressure.clone()

    want = project()
    relaxation = projector._jacobi if solver == 'JACOBI' else projector._relaxation
    assert relaxation.workspace is not None
    for look in (projector.metrics, projector.velocity_maxima, project):
        relaxation.workspace[:4].fill_(7)         # block 0 counts from another number
        projector.project(faces, out, 0.02)
        torch.cuda.synchronize()
        with pytest.raises(N.FfxError) as error:
            look()
        assert timed_out(error)
        assert torch.equal(project(), want)
        assert relaxation.timeouts() == 0
    projector.close()
