"""The collider multigrid's ways of running a solve against one another with whole
resident solves off, each shown to have run: the single-block tail, captured loops and
replayed cycles, the speculative sweep, fused sweeps. Same bits, cycles and sweeps.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def pair(shape, change, **settings):
    """Two projectors of one scene without resident solves; ``change`` acts on the second."""
    from tests.test_gpu_graph_resident import build
    (a, faces), (b, _) = build(shape, **settings), build(shape, **settings)
    for p in (a, b):
        p.use_resident = False
    change(b)
    return a, b, faces


def compare(a, b, faces, steps=3):
    out = [[torch.zeros_like(f) for f in faces] for _ in range(2)]
    for k in range(steps):
        scaled = [f * (1 + 0.3 * k) for f in faces]
        for p, o in zip((a, b), out):
            p.project(scaled, o, (0.02, 0.02, 0.01)[k % 3])
        assert a.last_cycles == b.last_cycles > 0
        assert a.last_iterations == b.last_iterations
        assert torch.equal(a.pressure, b.pressure)
        assert all(torch.equal(x, y) for x, y in zip(*out))
    assert a._coarse_resident() is None and b._coarse_resident() is None


@pytest.mark.parametrize('method,coarse', [('VCYCLE', 'DIRECT'), ('PCG', 'DIRECT'), ('VCYCLE', 'SMOOTH')])
@pytest.mark.parametrize('tolerance', [0.0, 1e-5])
def test_single_block_tail(method, coarse, tolerance):
    a, b, faces = pair((32, 32, 32), lambda p: setattr(p, 'use_tail', False), pressure_method=method,
                       coarse_solver=coarse, pressure_tolerance=tolerance, pressure_max_cycles=40, pressure_cycles=3)
    assert a.tail_start == 2 and len(a.levels) == 4
    compare(a, b, faces)
    a.close()
    b.close()


@pytest.mark.parametrize('method', ['VCYCLE', 'PCG', 'IR'])
def test_captured_against_eager(method):
    def eager(p):
        if method == 'IR':
            p.speculate = False     # (the refinement's loop is captured either way)
        else:
            p.use_graphs = False
    a, b, faces = pair((32, 24, 16), eager, pressure_method=method, pressure_tolerance=1e-5, pressure_max_cycles=60,
                       solid_warm_start=method == 'PCG')
    compare(a, b, faces)
    assert (a._graphs if method == 'PCG' else a._captured)
    if method != 'IR':
        assert not b._graphs and not b._captured
    a.close()
    b.close()


def test_replayed_cycles_of_a_fixed_budget():
    a, b, faces = pair((32, 24, 16), lambda p: setattr(p, 'use_graphs', False), pressure_cycles=3)
    compare(a, b, faces)
    assert a._graphs and not b._graphs
    a.close()
    b.close()


@pytest.mark.parametrize('shape', [(32, 32, 32), (64, 48, 40)])
@pytest.mark.parametrize('warm', [False, True])
def test_speculative_sweep(shape, warm):
    a, b, faces = pair(shape, lambda p: setattr(p, 'speculate', False), pressure_tolerance=1e-4,
                       pressure_max_cycles=40, solid_warm_start=warm)
    compare(a, b, faces)
    assert a._captured and b._captured
    a.close()
    b.close()


def test_device_loop_against_host_loop():
    a, b, faces = pair((48, 40, 32), lambda p: setattr(p, 'use_device_loop', False), pressure_tolerance=1e-4,
                       pressure_max_cycles=40)
    compare(a, b, faces)
    assert a._captured and not b._captured and b._graphs
    a.close()
    b.close()


def test_plans_of_whole_solves_are_no_captured_loops():
    from tests.test_gpu_graph_resident import build
    p, faces = build((32, 32, 32), pressure_tolerance=1e-4)
    p.project(faces, [torch.zeros_like(f) for f in faces], 0.02)
    assert p.last_cycles > 0 and not p._captured and not p._graphs
    assert list(p._loops) == ['resident'] and p._loops['resident'] is p._residents[0]
    p.close()
    assert not p._loops
