"""Device memory of an FP64 solver: what bounds the largest grid."""
import pytest

from afmibins_gb300 import capi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_fp64_solver_memory():
    """Velocity, its old copy, advection, right-hand sides, forces and scratch (18
    fields), divergence, two potentials and three CG vectors, and x, b and r on each
    level (8/7 of three): 27.4 fields of FP64, with 64 MB for the rest (walls, small
    levels, allocation granularity)."""
    with capi.Solver(16, mu=0.01, dt=1e-3):
        pass
    n = 192
    before = _free()
    with capi.Solver(n, mu=0.01, dt=1e-3):
        used = before - _free()
    assert used <= 8 * n ** 3 * (24 + 3 * 8 / 7) + (64 << 20)
