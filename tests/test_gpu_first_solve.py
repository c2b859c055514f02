"""A first solve finds its plan and workspace made and cleared, so it may be captured:
memory that a capture clears is clear in its replays only, and a solve outside them
would count its exchanges from whatever was there."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu


def projector_of(kind, shape, stream):
    from fluxfx_b200.backend.collision import SolidDevice, SolidPressureProjector
    from fluxfx_b200.backend.device import CudaDevice
    from fluxfx_b200.backend.multigrid import MultigridPressureProjector
    from fluxfx_b200.backend.pressure import PressureProjector
    from fluxfx_b200.backend.solid_multigrid import SolidMultigridProjector
    from fluxfx_b200.physics.collision import primitive
    from fluxfx_b200.physics.config import GridSpec
    from fluxfx_b200.physics.pressure import PressureSettings
    grid, device = GridSpec(shape), CudaDevice(stream=stream)
    if kind in ('masked', 'collider'):
        device = SolidDevice(grid, (primitive('SPHERE', (0.5, 0.5, 0.5), (0.2,) * 3),), device)
    make = dict(jacobi=PressureProjector, masked=SolidPressureProjector, geometric=MultigridPressureProjector,
                collider=SolidMultigridProjector)[kind]
    p = make(grid, PressureSettings(pressure_iterations=6), device)
    p.reset()
    g = torch.Generator(device='cuda').manual_seed(3)
    return p, [torch.rand(s[::-1], generator=g, device='cuda') - 0.5 for s in grid.face_shapes]


@pytest.mark.parametrize('kind,shape', [('jacobi', (32, 48, 40)), ('masked', (32, 48, 40)), ('geometric', (32, 48, 40)),
                                        ('geometric', (31, 23, 37)), ('collider', (31, 23, 37))])
def test_captured_first_solve(kind, shape):
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        p, faces = projector_of(kind, shape, side)
        out = [torch.zeros_like(f) for f in faces]
        p.project(faces, out, 0.02)
        want = p.pressure.clone()
        q, _ = projector_of(kind, shape, side)
        side.synchronize()
        gc.collect()                            # (as the capture does before it begins)
        held = torch.cuda.memory_allocated()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            q.project(faces, out, 0.02)
        assert torch.cuda.memory_allocated() - held <= 2048      # (the graph's own two words; a workspace has 100 KB)
        q.reset()
        q.project(faces, out, 0.02)            # outside the graph, before any replay
        assert torch.equal(q.pressure, want)
        for _ in range(2):
            q.pressure.zero_()
            graph.replay()
        side.synchronize()
        q.check_waits()
        p.close()
        q.close()
