"""Waits of resident solves that give up.

Blocks of a launch number their exchanges; a block whose stored number is altered
waits for words that never come, gives up after the bounded wait and runs to its
end, and so do its neighbours.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def build(**settings):
    from tests.test_gpu_graph_resident import build as make
    return make((32, 32, 32), **settings)


def solve(projector, rhs):
    """A whole solve of ``rhs`` from zero through the projector's plan."""
    from fluxfx_b200 import _native as N
    from fluxfx_b200.backend.device import ptr
    import torch
    plan = projector._resident(0)[0]
    p = torch.full_like(rhs, 7.0)
    tolerance = projector.settings.pressure_tolerance
    N.check(projector.device.lib.ffx_graph_solve(
        C.byref(plan), ptr(p), ptr(rhs), 0 if tolerance > 0 else 3, 1, tolerance, 9, ptr(projector._counters),
        projector.device.s))
    torch.cuda.synchronize()
    return p


def numbers(projector):
    """The plan's stored numbers (exchanges and decisions of every block): the words
    that its record at the workspace's start points to."""
    import torch
    _, workspace = projector._resident(0)
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
    projector.close()
