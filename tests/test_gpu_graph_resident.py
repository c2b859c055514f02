"""Resident collider solves (ffx_graph_solve) against the separate passes: bit for bit.

Shapes: two levels only (a coarsest level of 80 sweeps in tiles), a level that
stops halving at odd edges, rows that are no multiple of four, single-row tiles,
a direct coarsest level, a large one whose coarse part alone is resident.
"""
import ctypes as C

import pytest

from fluxfx_b200 import _native as N
from fluxfx_b200.backend.multigrid import hierarchy_shapes

SHAPES = [(16, 16, 16), (24, 20, 28), (34, 18, 22), (64, 32, 64), (48, 96, 48), (96, 80, 112), (32, 96, 96),
          (20, 64, 40)]
LARGE = [(160, 160, 112)]


def graph_plan(shapes, whole=True):
    plan = N.FfxGraphPlan()
    plan.count = len(shapes)
    plan.pre0 = plan.post0 = plan.pre = plan.post = 4
    plan.last_sweeps, plan.omega = 80, 2 / 3
    for k, s in enumerate(shapes):
        plan.level[k] = N.FfxGraphLevel(*s, None if k == 0 and whole else 4096, None, N.f3(1, 1, 1))
        if k == 0 and whole:
            plan.level[k].links = 4096      # planning looks at presence and alignment only
    return plan


@pytest.mark.parametrize('shape', SHAPES + LARGE)
def test_plans(shape):
    plan = graph_plan(hierarchy_shapes(shape))
    assert N.load().ffx_graph_plan(C.byref(plan)) == N.FFX_OK
    assert (plan.blocks > 0) == (shape in SHAPES)
    if plan.blocks:
        tiles = -(-shape[1] // plan.tile[0]) * -(-shape[2] // plan.tile[1])
        tail = plan.tail < plan.count
        assert plan.blocks == tiles + tail <= 148
        align = 2 ** (plan.tail if tail else plan.tail - 1)
        assert plan.tile[0] % align == 0 and plan.tile[1] % align == 0
    else:
        coarse = graph_plan(hierarchy_shapes(shape)[1:], whole=False)
        assert N.load().ffx_graph_plan(C.byref(coarse)) == N.FFX_OK and coarse.blocks > 0


def build(shape, **settings):
    import torch
    from fluxfx_b200.backend.collision import SolidDevice
    from fluxfx_b200.backend.solid_multigrid import SolidMultigridProjector
    from fluxfx_b200.physics.collision import primitive
    from fluxfx_b200.physics.config import GridSpec
    from fluxfx_b200.physics.pressure import PressureSettings
    extent = tuple(n / max(shape) for n in shape)
    grid = GridSpec(shape, extent, axis_limit=max(128, *shape))
    r = 0.21 * min(extent)
    colliders = (primitive('SPHERE', tuple(0.52 * e for e in extent), (r,) * 3),
                 primitive('BOX', tuple(0.2 * e for e in extent), tuple(0.13 * e for e in extent)))
    device = SolidDevice(grid, colliders)
    projector = SolidMultigridProjector(grid, PressureSettings(**settings), device)
    projector.reset()
    g = torch.Generator(device='cuda').manual_seed(sum(shape))
    faces = [torch.rand(s[::-1], generator=g, device='cuda') - 0.5 for s in grid.face_shapes]
    return projector, faces


@pytest.mark.gpu
@pytest.mark.parametrize('shape', SHAPES + LARGE)
@pytest.mark.parametrize('settings', [
    dict(), dict(pressure_tolerance=1e-3, pressure_max_cycles=12),
    dict(pressure_tolerance=1e-4, pressure_max_cycles=20, solid_warm_start=True, mg_coarse_scale=1.7,
         mg_pre_sweeps=2, mg_post_sweeps=2, mg_coarse_sweeps=3)])
def test_bit_identical_to_the_separate_passes(shape, settings):
    import torch
    results = []
    for resident in (True, False):
        projector, faces = build(shape, **settings)
        projector.use_resident = resident
        out = [torch.zeros_like(f) for f in faces]
        seen = []
        for step in range(3):
            projector.project([f * (1 + 0.1 * step) for f in faces], out, 0.02)
            seen.append((projector.last_cycles, projector.last_iterations, projector.pressure.clone(),
                         [o.clone() for o in out]))
        assert projector.resident_timeouts() == 0
        assert bool(projector._residents.get(0) or projector._residents.get(1)) == resident
        results.append((seen, projector.total_cycles()))
        projector.close()
    (a, total_a), (b, total_b) = results
    assert total_a == total_b
    for (ca, ia, pa, oa), (cb, ib, pb, ob) in zip(a, b):
        assert (ca, ia) == (cb, ib)
        assert torch.equal(pa, pb) and all(torch.equal(x, y) for x, y in zip(oa, ob))


@pytest.mark.gpu
def test_zero_right_hand_side_and_converged_start():
    import torch
    projector, faces = build((48, 40, 56), pressure_tolerance=1e-3, solid_warm_start=True)
    out = [torch.zeros_like(f) for f in faces]
    projector.project(faces, out, 0.02)
    kept = projector.pressure.clone()
    projector.project(faces, out, 0.02)                # the start already meets the tolerance
    assert projector.last_cycles == 0 and torch.equal(projector.pressure, kept)
    projector.project([torch.zeros_like(f) for f in faces], out, 0.02)
    assert projector.last_cycles == 0 and not bool(projector.pressure.any())
    assert projector.resident_timeouts() == 0
