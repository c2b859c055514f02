"""Whole relaxation solves (``backend/relax.py``) against the FP64 oracle's sweeps and cycles.

Tolerance: a sweep rounds each cell's update some eight times, and weighted
Jacobi does not amplify earlier errors, so after n sweeps a cell is at most
about 8 n roundings of the largest pressure off; a V-cycle adds its coarse
levels' sweeps and its transfers. The bound used is 8 (n + 16) 2^-24 max|p|
with n all sweeps of all levels.
"""
import ctypes as C

import numpy as np
import pytest

from fluxfx_b200 import _native as N
from fluxfx_b200.backend.multigrid import hierarchy_shapes
from fluxfx_b200.physics.coarse_pressure import neumann_basis, neumann_inverse
from oracle import smoke as S

# grids that one block holds, that tiles hold (ragged, rim-only and odd tiles, both copies of the
# pressure, the largest), and that are relaxed a few sweeps per launch
RESIDENT = [(2, 2, 2), (16, 16, 16), (32, 32, 32), (75, 61, 93), (33, 2, 70), (127, 9, 5), (128, 128, 128),
            (128, 96, 112), (45, 30, 35), (160, 96, 100), (130, 24, 24)]
LARGE = [(256, 128, 64), (301, 70, 93)]


def bound(n, p):
    return 8 * (n + 16) * 2.0 ** -24 * float(np.abs(p).max())


def extent_of(shape):
    return tuple(n / max(shape) * 1.25 for n in shape)


def plan_of(shapes, extent, classes=False):
    plan = N.FfxRelaxPlan()
    plan.count, plan.pre, plan.post, plan.last_sweeps, plan.omega = len(shapes), 3, 3, 80, 2 / 3
    plan.classes = 4 if classes else None      # planning looks at its presence only
    for slot, shape in zip(plan.level, shapes):
        slot.grid = N.FfxRelaxGrid(N.n3(*shape), N.f3(*[n / e for n, e in zip(shape, extent)]))
    return plan


@pytest.mark.parametrize('shape', RESIDENT + LARGE)
def test_every_grid_gets_a_plan(shape):
    for shapes in ([shape], hierarchy_shapes(shape)):
        plan = plan_of(shapes, extent_of(shape))
        assert N.load().ffx_relax_plan(C.byref(plan)) == N.FFX_OK
        resident = plan.tail == 0 or plan.tile[0] > 0
        assert resident == (shape in RESIDENT)
        if resident and plan.tail:
            tiles = -(-shape[1] // plan.tile[0]) * -(-shape[2] // plan.tile[1])
            assert tiles + (plan.tail < plan.count) <= 148
            align = 2 ** (plan.tail if plan.tail < plan.count else plan.tail - 1)
            assert plan.tile[0] % align == 0 and plan.tile[1] % align == 0


@pytest.mark.parametrize('shape', [(4, 4, 4), (8, 8, 8), (4, 8, 16), (6, 5, 7)])
def test_separable_basis_is_the_dense_inverse(shape):
    extent = (1.0, 0.8, 1.3)
    v = neumann_basis(shape, extent)
    parts = np.split(v, np.cumsum([n * n for n in shape]))
    bx, by, bz = (p.reshape(n, n) for p, n in zip(parts, shape))
    r = np.random.default_rng(1).normal(size=shape[::-1])
    modes = np.einsum('ia,jb,kc,cba->kji', bx, by, bz, r) * parts[3].reshape(shape[::-1])
    got = np.einsum('ia,jb,kc,kji->cba', bx, by, bz, modes)
    want = (neumann_inverse(shape, extent) @ r.ravel()).reshape(r.shape)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()


def oracle_grid(shape, mask=None):
    return S.Grid(shape, extent_of(shape), np.float64, mask=mask)


def fields(shape, seed):
    rng = np.random.default_rng(seed)
    rhs = rng.normal(size=shape[::-1])
    return (rhs - rhs.mean()).astype(np.float32), rng.normal(size=shape[::-1]).astype(np.float32) * 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize('shape', RESIDENT + LARGE)
@pytest.mark.parametrize('masked', [False, True])
def test_sweeps(shape, masked):
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.relax import Relaxation
    dev = CudaDevice()
    rhs, p0 = fields(shape, 3)
    mask = (np.random.default_rng(4).random(shape[::-1]) < 0.2) if masked else None
    g = oracle_grid(shape, mask)
    classes = None
    if masked:
        nx, ny, nz = shape
        classes = torch.empty((nz, ny, (nx + 3) // 4 * 4), dtype=torch.uint8, device='cuda')
        solid = torch.as_tensor(mask.astype(np.uint8)).cuda()
        dev.call('ffx_relax_classes', N.n3(*shape), C.c_void_p(solid.data_ptr()), C.c_void_p(classes.data_ptr()),
                 dev.s)
    r = Relaxation(dev, [shape], extent_of(shape), 0.6, last=11, classes=classes)
    for from_zero, dt in ((True, 1.0), (False, 0.04)):
        p, q = torch.as_tensor(p0).cuda(), torch.zeros(shape[::-1], device='cuda')
        got, _ = r.run(p, q, torch.as_tensor(rhs).cuda(), 1, dt, from_zero)
        want = np.zeros_like(p0, dtype=np.float64) if from_zero else p0.astype(np.float64)
        for _ in range(11):
            want = S.jacobi(g, want, rhs.astype(np.float64), dt, 0.6, mask=mask)
        assert np.abs(got.double().cpu().numpy() - want).max() <= bound(11, want)
    assert r.timeouts() == 0


@pytest.mark.gpu
@pytest.mark.parametrize('shape,levels,sweeps', [((8, 8, 8), 0, 3), ((16, 16, 16), 0, 3), ((32, 32, 32), 0, 3),
                                                 ((64, 64, 64), 4, 2), ((64, 64, 64), 0, 16), ((16, 64, 32), 0, 1),
                                                 ((128, 96, 112), 0, 3), ((128, 128, 128), 0, 3), ((90, 60, 70), 0, 3),
                                                 ((44, 20, 120), 0, 3), ((160, 96, 96), 0, 3), ((256, 128, 64), 0, 9),
                                                 ((264, 72, 88), 0, 3)])
def test_cycles(shape, levels, sweeps):
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.relax import Relaxation
    dev = CudaDevice()
    shapes = hierarchy_shapes(shape, levels)
    direct = shapes[-1] == (4, 4, 4) or levels
    extent = extent_of(shape)
    basis = torch.as_tensor(neumann_basis(shapes[-1], extent)).cuda() if direct else None
    r = Relaxation(dev, shapes, extent, 2 / 3, pre=sweeps, post=sweeps, last=80, basis=basis)
    mg = S.GeometricMG(oracle_grid(shape), sweeps, sweeps, levels,
                       neumann_inverse(shapes[-1], extent) if direct else None)
    rhs, p0 = fields(shape, 5)
    n = 2 * (2 * sweeps * (len(shapes) - 1) + (0 if direct else 80))
    for from_zero, dt in ((True, 1.0), (False, 0.04)):
        p, q = torch.as_tensor(p0).cuda(), torch.zeros(shape[::-1], device='cuda')
        want = np.zeros_like(p0, dtype=np.float64) if from_zero else p0.astype(np.float64)
        for _ in range(2):
            want = mg.cycle(0, want, rhs.astype(np.float64), dt)
        rhs_t = torch.as_tensor(rhs).cuda()
        got, _ = r.run(p, q, rhs_t, 2, dt, from_zero)
        assert np.abs(got.double().cpu().numpy() - want).max() <= bound(n, want)
        # the same two cycles one call at a time
        a, b = torch.as_tensor(p0).cuda(), torch.zeros(shape[::-1], device='cuda')
        a, b = r.run(a, b, rhs_t, 1, dt, from_zero)
        a, b = r.run(a, b, rhs_t, 1, dt, False)
        assert torch.equal(a, got)
    assert r.timeouts() == 0


@pytest.mark.gpu
def test_resident_solve_under_capture():
    """A captured solve replays: the exchanges' numbers live on the device."""
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.relax import Relaxation
    shape = (48, 40, 56)
    rhs, p0 = fields(shape, 6)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        dev = CudaDevice(stream=side)
        r = Relaxation(dev, [shape], extent_of(shape), 2 / 3, last=5)
        p, q, f = torch.as_tensor(p0).cuda(), torch.zeros(shape[::-1], device='cuda'), torch.as_tensor(rhs).cuda()
        want = p.clone()
        for _ in range(4):
            r.run(want, q, f, 1, 1.0, False)
        graph = torch.cuda.CUDAGraph()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            r.run(p, q, f, 1, 1.0, False)
        for _ in range(4):
            graph.replay()
        side.synchronize()
    assert torch.equal(p, want) and r.timeouts() == 0


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_counted():
    """Blocks that expect different exchange numbers give up after the limit and say so."""
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.relax import Relaxation
    shape = (32, 32, 32)
    r = Relaxation(CudaDevice(), [shape], (1.0, 1.0, 1.0), 2 / 3, last=1)
    p, q, f = (torch.zeros(shape[::-1], device='cuda') for _ in range(3))
    r.run(p, q, f, 1, 1.0, False)
    assert r.timeouts() == 0
    r.workspace[:4].fill_(7)       # block 0 counts from another number than its neighbours
    r.run(p, q, f, 1, 1.0, False)
    assert r.timeouts() > 0
