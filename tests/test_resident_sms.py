"""Plans of resident solves on fewer SMs than a whole chip has: they use no more
blocks than they are given, and what does not fit takes the launches that need no
co-residency. ``sms`` 1 is what a device without cooperative launches reports.
"""
import ctypes as C

import numpy as np
import pytest

from fluxfx_b200 import _native as N
from fluxfx_b200.backend.multigrid import hierarchy_shapes
from tests.test_gpu_graph_resident import graph_plan
from tests.test_gpu_relax import bound, extent_of, fields, oracle_grid, plan_of

SMS = [1, 2, 20, 74, 132, 148, 0]


@pytest.mark.parametrize('sms', SMS)
@pytest.mark.parametrize('shape', [(16, 16, 16), (32, 32, 32), (75, 61, 93), (128, 96, 112), (128, 128, 128)])
def test_relaxation_plans(shape, sms):
    for shapes in ([shape], hierarchy_shapes(shape)):
        for classes in (False, True)[:1 + (len(shapes) == 1)]:
            plan = plan_of(shapes, extent_of(shape), classes)
            plan.sms = sms
            assert N.load().ffx_relax_plan(C.byref(plan)) == N.FFX_OK
            assert plan.sms == (sms or 148)
            if plan.tail and plan.tile[0]:
                tiles = -(-shape[1] // plan.tile[0]) * -(-shape[2] // plan.tile[1])
                assert tiles + (plan.tail < plan.count) <= plan.sms
            elif plan.tail:      # several sweeps per launch: every level above the tail has its tiles
                assert all(plan.level[k].sweep.sweeps >= 1 for k in range(plan.tail))
            if sms == 1:
                assert plan.tail == 0 or not plan.tile[0] or plan.tile[0] >= shape[1] and plan.tile[1] >= shape[2]


@pytest.mark.parametrize('sms', SMS)
@pytest.mark.parametrize('shape', [(16, 16, 16), (48, 96, 48), (96, 80, 112), (160, 160, 112)])
def test_collider_plans(shape, sms):
    for whole in (True, False):
        plan = graph_plan(hierarchy_shapes(shape)[0 if whole else 1:], whole)
        plan.sms = sms
        assert N.load().ffx_graph_plan(C.byref(plan)) == N.FFX_OK
        assert plan.blocks <= plan.sms == (sms or 148)
        if sms == 1:
            assert plan.blocks == 0


@pytest.mark.gpu
@pytest.mark.parametrize('sms', [1, 20, 74])
@pytest.mark.parametrize('shape', [(32, 32, 32), (75, 61, 93)])
def test_sweeps_and_cycles_on_fewer_sms(shape, sms):
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.relax import Relaxation
    from oracle import smoke as S
    dev = CudaDevice()
    rhs, p0 = fields(shape, 8)
    g = oracle_grid(shape)
    r = Relaxation(dev, [shape], extent_of(shape), 0.6, last=9, sms=sms)
    p, q = torch.as_tensor(p0).cuda(), torch.zeros(shape[::-1], device='cuda')
    got, _ = r.run(p, q, torch.as_tensor(rhs).cuda(), 1, 0.04, False)
    want = p0.astype(np.float64)
    for _ in range(9):
        want = S.jacobi(g, want, rhs.astype(np.float64), 0.04, 0.6)
    assert np.abs(got.double().cpu().numpy() - want).max() <= bound(9, want)
    shapes = hierarchy_shapes(shape)
    if len(shapes) == 1:
        return
    whole, fewer = (Relaxation(dev, shapes, extent_of(shape), 2 / 3, pre=3, post=3, last=80, sms=n) for n in (0, sms))
    fields_t = [torch.as_tensor(f).cuda() for f in (p0, np.zeros_like(p0), rhs)]
    a, _ = whole.run(*[f.clone() for f in fields_t], 2, 0.04, False)
    b, _ = fewer.run(*[f.clone() for f in fields_t], 2, 0.04, False)
    n = 2 * (6 * (len(shapes) - 1) + 80)
    assert np.abs((a - b).double().cpu().numpy()).max() <= 2 * bound(n, a.double().cpu().numpy())
    assert r.timeouts() == whole.timeouts() == fewer.timeouts() == 0


@pytest.mark.gpu
@pytest.mark.parametrize('sms', [40, 74])
def test_collider_solve_on_fewer_sms(sms):
    """Other tiles, the same bits."""
    import torch
    from fluxfx_b200.backend.device import ptr
    from tests.test_gpu_graph_resident import build
    projector, _ = build((64, 32, 64))
    dev = projector.device
    generator = torch.Generator(device='cuda').manual_seed(4)
    rhs = torch.randn(projector.before.shape, generator=generator, device='cuda')
    results = []
    for n in (0, sms):
        plan = N.FfxGraphPlan.from_buffer_copy(projector._resident(0)[0])
        plan.sms, plan.alarm = n, None
        N.check(dev.lib.ffx_graph_plan(C.byref(plan)))
        assert 0 < plan.blocks <= (n or 148)
        workspace = torch.zeros(plan.workspace_bytes, dtype=torch.uint8, device='cuda')
        plan.workspace = workspace.data_ptr()
        N.check(dev.lib.ffx_graph_plan_upload(C.byref(plan), dev.s))
        p = torch.zeros_like(rhs)
        N.check(dev.lib.ffx_graph_solve(C.byref(plan), ptr(p), ptr(rhs), 3, 1, 0.0, 0, None, dev.s))
        torch.cuda.synchronize()
        results.append(p)
    assert torch.equal(*results)
    projector.close()
