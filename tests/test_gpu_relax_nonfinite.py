"""Infinities and NaNs in a relaxation solve reach the cells that single sweeps
(``ffx_jacobi``) carry them to and no others: walls hold them, and so do the ends
of rows that are no multiple of four.

Every other cell has finite neighbours only, so it keeps the bound of the solves
against the sweeps: 8 (n + 16) 2^-24 max|p| for either after n sweeps.
"""
import ctypes as C

import numpy as np
import pytest

from fluxfx_b200 import _native as N

pytestmark = pytest.mark.gpu


def solves(shape, solid, rhs, p0, dt, from_zero, sweeps):
    """The iterate by one solve and by single sweeps."""
    import torch
    from fluxfx_b200.backend.device import CudaDevice, ptr
    from fluxfx_b200.backend.relax import Relaxation
    dev = CudaDevice()
    nx, ny, nz = shape
    extent = tuple(n / max(shape) for n in shape)
    mask = classes = None
    if solid is not None:
        mask = torch.as_tensor(solid.astype(np.uint8)).cuda()
        classes = torch.empty((nz, ny, (nx + 3) // 4 * 4), dtype=torch.uint8, device='cuda')
        dev.call('ffx_relax_classes', N.n3(*shape), ptr(mask), ptr(classes), dev.s)
    f = torch.as_tensor(rhs).cuda()
    r = Relaxation(dev, [shape], extent, 2 / 3, last=sweeps, classes=classes)
    p, q = torch.as_tensor(p0).cuda(), torch.zeros(shape[::-1], device='cuda')
    got, _ = r.run(p, q, f, 1, dt, from_zero)
    a = torch.zeros_like(q) if from_zero else torch.as_tensor(p0).cuda()
    b = torch.empty_like(a)
    inv = N.f3(*[n / e for n, e in zip(shape, extent)])
    for _ in range(sweeps):
        dev.call('ffx_jacobi', N.n3(*shape), inv, ptr(mask), ptr(a), ptr(f), dt, 2 / 3, ptr(b), dev.s)
        a, b = b, a
    assert r.timeouts() == 0
    return got.double().cpu().numpy(), a.double().cpu().numpy()


# tiles with one and two copies of the pressure, ragged rows, and several sweeps per launch
SHAPES = [(24, 20, 28), (75, 61, 93), (127, 9, 50), (128, 128, 128), (301, 70, 93)]


@pytest.mark.parametrize('shape', SHAPES)
@pytest.mark.parametrize('walled', [False, True])
@pytest.mark.parametrize('from_zero', [True, False])
def test_non_finite_values_stay_where_single_sweeps_keep_them(shape, walled, from_zero):
    nx, ny, nz = shape
    rng = np.random.default_rng(9)
    rhs = rng.normal(size=shape[::-1]).astype(np.float32)
    p0 = rng.normal(size=shape[::-1]).astype(np.float32) * 1e-3
    solid = None
    if walled:
        solid = np.zeros(shape[::-1], bool)
        solid[nz // 2] = solid[:, ny // 2] = True        # four chambers
        rhs[nz // 2, 2, 3] = np.inf                      # inside the wall: never read
        p0[0, ny // 2, nx - 1] = np.nan
    # beside the walls, at a row's end, in different chambers; one chamber stays clean
    rhs[nz // 2 - 1, 1, nx - 1] = np.nan
    rhs[nz // 2 + 1, ny // 2 - 1, nx // 2] = np.inf
    rhs[nz // 2 + 1, ny // 2 - 1, nx // 2 - 1] = -np.inf
    sweeps = 11
    got, want = solves(shape, solid, rhs, p0, 0.04, from_zero, sweeps)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert 0 < np.count_nonzero(~np.isfinite(want)) < want.size // 2
    keep = np.isfinite(want)
    bound = 2 * 8 * (sweeps + 16) * 2.0 ** -24 * np.abs(want[keep]).max()
    assert np.abs(got[keep] - want[keep]).max() <= bound
    if walled:
        assert not got[solid].any() and np.isfinite(got[:nz // 2, ny // 2:]).all()


@pytest.mark.parametrize('shape', [(32, 32, 32), (30, 32, 32), (28, 24, 40), (128, 96, 112)])
def test_whole_cycles_beside_padding(shape):
    """A V-cycle's smoothing on a level whose rows end in padding (level 0, or a coarse
    one below whole float4): what is not finite stays off the cells that no sweep,
    transfer or coarse solve has carried it to, which with a direct or 80-sweep coarsest
    level are none, so every cell becomes NaN or infinite, and a clean right-hand side
    gives a finite pressure in the next solve of the same workspace."""
    import torch
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.multigrid import hierarchy_shapes
    from fluxfx_b200.backend.relax import Relaxation
    r = Relaxation(CudaDevice(), hierarchy_shapes(shape), tuple(n / max(shape) for n in shape), 2 / 3, pre=3, post=3,
                   last=80)
    g = torch.Generator(device='cuda').manual_seed(1)
    f = torch.randn(shape[::-1], generator=g, device='cuda')
    p, q = torch.zeros_like(f), torch.zeros_like(f)
    want = r.run(p, q, f, 2, 1.0, True)[0].clone()
    bad = f.clone()
    bad[shape[2] // 2, 1, shape[0] - 1] = float('nan')
    assert not bool(torch.isfinite(r.run(p, q, bad, 1, 1.0, True)[0]).any())
    assert torch.equal(r.run(p, q, f, 2, 1.0, True)[0], want) and bool(torch.isfinite(want).all())
    assert r.timeouts() == 0
