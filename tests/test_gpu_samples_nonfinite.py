"""Samples beside values that are not finite.

A coordinate clamped to the last sample of an axis reads that one alone: a NaN or
an infinity in the sample before it has no part (mac_sample.glsl:2-19 clamps both
corners). A corner that is infinite and has a weight gives an infinity, not a NaN.
There the oracle, which evaluates the shaders' operations, is the measure, with
the suite's bound for finite results.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import smoke as S
from tests.gpu_helpers import assert_close, dev, grid_ptr, n, solids, t
from tests.test_gpu_passes import ptr

pytestmark = pytest.mark.gpu

# powers of two and ragged sizes: the forms of the sampler's positions
GRIDS = [((8, 4, 16), (0.5, 0.25, 1.0)), ((33, 9, 6), (1.1, 0.3, 0.2)), ((37, 35, 34), (0.9, 0.8, 0.7))]


@pytest.mark.parametrize('shape,extent', GRIDS)
@pytest.mark.parametrize('storage', ['FP32', 'BF16'])
@pytest.mark.parametrize('bad', [np.nan, np.inf])
def test_the_last_sample_counts_alone(shape, extent, storage, bad):
    D = dev()
    _, gp = grid_ptr(shape, extent)
    so = solids()
    dtype, code = (torch.float32, 0) if storage == 'FP32' else (torch.bfloat16, 1)
    dt = 0.9 * min(e / k for e, k in zip(extent, shape))     # a trace of less than a cell
    faces = S.Grid(shape, extent).face_shapes
    for axis in range(3):
        for component in range(3):
            # a uniform flow whose traces go out of the domain at the upper wall of
            # `axis`; the samples before the last along it are not finite
            value = [-0.75 if c == axis else 0.25 for c in range(3)]
            vel = [np.full(fs, v, np.float32) for fs, v in zip(faces, value)]
            along = 2 - axis
            np.moveaxis(vel[component], along, 0)[-2] = bad
            outs = [t(np.zeros(fs), dtype) for fs in faces]
            D.call('ffx_face_predictor', gp, C.byref(so), code, *[ptr(t(v, dtype)) for v in vel], dt,
                   *map(ptr, outs), D.s)
            got = np.moveaxis(n(outs[component]), along, 0)[-1]
            # (the uniform value, to the rounding of a sample's eight weights)
            assert np.abs(got - value[component]).max() <= 2.0 ** -20, (axis, component)


@pytest.mark.parametrize('shape,extent', GRIDS)
@pytest.mark.parametrize('masked', [False, True])
def test_an_infinity_with_a_weight_stays_one(shape, extent, masked):
    D = dev()
    mask = np.zeros(shape[::-1], np.uint8)
    g = S.Grid(shape, extent, mask=mask.astype(bool) if masked else None)
    _, gp = grid_ptr(shape, extent)
    so = solids(t(mask, torch.uint8), t(mask, torch.uint8)) if masked else solids()
    # a uniform flow: every fraction lies well inside (0, 1)
    h = [e / k for e, k in zip(extent, shape)]
    dt = 0.5 * min(h)
    vel = [np.full(fs, 0.4 * w / dt, np.float32) for w, fs in zip(h, g.face_shapes)]
    field = np.random.default_rng(2).uniform(0, 1, g.cell_shape).astype(np.float32)
    z, y, x = (k // 2 for k in field.shape)
    field[z, y, x] = np.inf
    field[0, 0, 0] = -np.inf
    field[-1, -1, 1] = np.nan
    field_t, out = t(field), t(np.zeros(g.cell_shape))
    D.call('ffx_scalar_transport', gp, C.byref(so), 0, *[ptr(t(v)) for v in vel], dt, 1,
           (C.c_void_p * 1)(field_t.data_ptr()), (C.c_void_p * 1)(out.data_ptr()), D.s)
    with np.errstate(all='ignore'):
        want = S.scalar_transport(g, vel, field, dt)
    got = n(out)
    assert np.isinf(want).sum() >= 8
    for kind in (np.isposinf, np.isneginf, np.isnan):
        assert np.array_equal(kind(got), kind(want)), kind
    keep = np.isfinite(want)
    assert_close(got[keep], want[keep])
