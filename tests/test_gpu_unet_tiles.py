"""Convolutions at the edges of their tiles: up-samplings whose input voxels end
inside a block, every channel count of the per-voxel kernels, and few rows with
more channels than a block takes (narrower blocks, the last one partly empty).

Tolerance: K products of BF16 values are exact in FP32 and summed in FP32, so a
result lies within K 2^-23 sum |products| of the FP64 one.
"""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from fluxfx_b200 import _native as N
from tests.test_gpu_unet import bf, conv_struct

pytestmark = pytest.mark.gpu


def formed(kind, x, w):
    """FP64 result and sum of |products| (channels last)."""
    out = []
    for a, b in ((x.double(), w.double()), (x.double().abs(), w.double().abs())):
        a = a.permute(0, 4, 1, 2, 3)
        if kind == 'up':
            k = b.view(2, 2, 2, *b.shape[1:]).permute(3, 4, 0, 1, 2)
            r = F.conv_transpose3d(a, k, stride=2)
        else:
            k = b.view(2, 2, 2, *b.shape[1:]).permute(4, 3, 0, 1, 2)
            r = F.conv3d(a, k, stride=2)
        out.append(r.permute(0, 2, 3, 4, 1))
    return out


@pytest.mark.parametrize('kind,batch,small,cin,cout,entry', [
    ('up', 1, (1, 1, 1), 8, 8, 'ffx_conv_forward_tma'), ('up', 2, (7, 5, 9), 24, 16, 'ffx_conv_forward_tma'),
    ('up', 1, (4, 8, 8), 64, 8, 'ffx_conv_forward_tma'), ('up', 1, (3, 3, 29), 96, 16, 'ffx_conv_forward_tma'),
    ('up', 2, (3, 5, 7), 48, 40, 'ffx_conv_forward'), ('up', 1, (5, 4, 13), 128, 64, 'ffx_conv_forward'),
    ('down', 1, (2, 3, 5), 16, 72, 'ffx_conv_forward'), ('down', 2, (4, 4, 9), 40, 64, 'ffx_conv_forward'),
    ('down', 1, (1, 1, 1), 8, 32, 'ffx_conv_forward')])
def test_convolutions_at_tile_edges(kind, batch, small, cin, cout, entry):
    lib = N.load()
    g = torch.Generator().manual_seed(cin + cout)
    large = tuple(2 * v for v in small)
    ind, outd = (small, large) if kind == 'up' else (large, small)
    x = bf(torch.randn((batch, *ind, cin), generator=g))
    w = bf(torch.randn((8, cin, cout), generator=g))
    dx, dw, out = x.cuda(), w.cuda(), torch.full((batch, *outd, cout), 7., device='cuda')
    c = conv_struct(batch, ind, outd, cin, 0, cout, 2, 2, 0, int(kind == 'up'), dx, cin, 0, None, 0, 0, dw, None, 0,
                    None, 0, 0, out, cout)
    args = (C.byref(c), None, None) if entry == 'ffx_conv_forward_tma' else (C.byref(c), None)
    N.check(getattr(lib, entry)(*args))
    torch.cuda.synchronize()
    ref, size = formed(kind, x, w)
    K = cin * (1 if kind == 'up' else 8)
    assert bool(((out.cpu().double() - ref).abs() <= K * 2.0 ** -23 * size + 1e-30).all())
