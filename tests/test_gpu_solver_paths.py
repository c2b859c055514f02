"""Where the collider multigrid keeps what its solves run on."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_plans_of_whole_solves_are_no_captured_loops():
    from tests.test_gpu_graph_resident import build
    p, faces = build((32, 32, 32), pressure_tolerance=1e-4)
    p.project(faces, [torch.zeros_like(f) for f in faces], 0.02)
    assert p.last_cycles > 0 and not p._captured and not p._graphs
    assert list(p._loops) == ['resident'] and p._loops['resident'] is p._residents[0]
    p.close()
    assert not p._loops
