"""Transport passes at the edges of their samples and tiles: axes of one cell
(one sample on both sides), rows of whole 32-cell tiles (the last column's faces
share tiles), traces that leave the domain (clamped corners), 16-bit storage.

Tolerance without colliders: a grid coordinate formed as p (n/e) lies within
delta = 2^-22 max(n) cells of the oracle's p n / e; a sample of fields of size m
then within 6 delta m (three axes, slopes up to 2 m), a trace of D cells moves by
D times that at its midpoint and again at its end: 6 delta (1 + 6 D + 18 D^2) m.
With colliders the operations are the oracle's: the suite's own bound.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import smoke as S
from tests.gpu_helpers import REL, assert_close, dev, grid_ptr, n, random_faces, solids, t
from tests.test_gpu_passes import _mask_setup, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(1, 6, 5), (5, 1, 4), (4, 3, 1), (2, 2, 2), (32, 5, 4), (64, 258, 3), (33, 9, 6)])
@pytest.mark.parametrize('cells', [0.6, 5.0])
@pytest.mark.parametrize('masked', [False, True])
def test_traces_match_oracle(shape, cells, masked):
    D = dev()
    rng = np.random.default_rng(5)
    extent = tuple(0.9 * v / max(shape) for v in shape)
    mask, halo = _mask_setup(D, shape, extent) if masked else (None, None)
    g = S.Grid(shape, extent, mask=n(mask).astype(bool) if masked else None)
    _, gp = grid_ptr(shape, extent)
    so = solids(mask, halo)
    vel = random_faces(g, rng, 1.0)
    vel_t = [t(v) for v in vel]
    dt = cells * 0.9 / max(shape)
    delta = 2.0 ** -22 * max(shape)
    rel = REL if masked else max(REL, 6 * delta * (1 + 6 * cells + 18 * cells ** 2))
    faces = [t(np.zeros(fs)) for fs in g.face_shapes]
    D.call('ffx_face_predictor', gp, C.byref(so), 0, *map(ptr, vel_t), dt, *map(ptr, faces), D.s)
    for a in range(3):
        assert_close(n(faces[a]), S.face_predictor(g, vel, a, dt), rel=rel, what=f'faces {a}')
    field = rng.uniform(0, 1, g.cell_shape).astype(np.float32)
    if masked:
        field = np.where(g.mask, 0, field).astype(np.float32)
    field_t, out = t(field), t(np.zeros(g.cell_shape))
    D.call('ffx_scalar_transport', gp, C.byref(so), 0, *map(ptr, vel_t), dt, 1, (C.c_void_p * 1)(field_t.data_ptr()),
           (C.c_void_p * 1)(out.data_ptr()), D.s)
    expected = S.scalar_transport(g, vel, field, dt)
    assert_close(n(out), expected, rel=rel, what='scalar')
    # 16-bit storage of the same values: its rounding of inputs (2^-9 of a value, on
    # velocities too) and of the result
    if cells < 1 and not masked:
        vel_16 = [t(v).to(torch.bfloat16) for v in vel]
        field_16, out_16 = field_t.to(torch.bfloat16), torch.zeros_like(field_t, dtype=torch.bfloat16)
        D.call('ffx_scalar_transport', gp, C.byref(so), 1, *map(ptr, vel_16), dt, 1,
               (C.c_void_p * 1)(field_16.data_ptr()), (C.c_void_p * 1)(out_16.data_ptr()), D.s)
        rounded = S.scalar_transport(g, [v.float().cpu().numpy() for v in vel_16], field_16.float().cpu().numpy(), dt)
        assert_close(out_16.float().cpu().numpy(), rounded, rel=rel + 2.0 ** -8, what='16-bit scalar')
