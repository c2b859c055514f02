"""Resident solves of several domains issued on their own streams at once: each
launch has all its blocks on the chip or none, so they queue behind one another
and give the results of solves issued one by one, with no wait given up."""
import pytest
import torch

from tests.test_gpu_graph_resident import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shapes', [[(48, 96, 48), (96, 80, 112), (64, 32, 64), (24, 20, 28)]])
def test_concurrent_streams(shapes):
    import ctypes as C

    from fluxfx_b200 import _native as N
    from fluxfx_b200.backend.device import ptr
    projectors = [build(s)[0] for s in shapes]
    for k, p in enumerate(projectors):
        p.before.copy_(torch.randn(p.before.shape, generator=torch.Generator().manual_seed(k)))

    def solve(p, stream):
        plan = p._resident(0)[0]
        N.check(p.device.lib.ffx_graph_solve(C.byref(plan), ptr(p.pressure), ptr(p.before), 2, 1, 0.0, 0, None, stream))

    expected = []
    for p in projectors:
        solve(p, p.device.s)
        torch.cuda.synchronize()
        expected.append(p.pressure.clone())
    streams = [torch.cuda.Stream() for _ in projectors]
    torch.cuda.synchronize()
    for _ in range(25):
        for p, s in zip(projectors, streams):
            solve(p, C.c_void_p(s.cuda_stream))
    torch.cuda.synchronize()
    for p, e in zip(projectors, expected):
        assert p.resident_timeouts() == 0
        assert torch.equal(p.pressure, e)
