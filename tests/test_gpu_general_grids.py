"""Grids whose extents are not powers of two on the batched kernels and the
interleaved double-float viscous solves."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _steps(dims, bc, precision):
    n = 40
    g = po.Grid(*dims, n, channel=bc == capi.BC_CHANNEL)
    rng = np.random.default_rng(31)
    u, v, w = (0.1 * rng.standard_normal(k) for k in (g.ncell, g.nv, g.ncell))
    f = [rng.standard_normal(k) for k in (g.ncell, g.nv, g.ncell)]
    with capi.Solver(*dims, n=n, bc=bc, precision=precision, mu=0.01, rho=1.0, dt=1e-3, tol=TOL) as sv:
        sv.set_velocity(u, v, w)
        sv.project()
        for _ in range(3):
            sv.ns_step(*f)
        return sv.get_velocity(), sv.stats()["outer_iters"]


@pytest.mark.parametrize("dims", [(40, 24, 16), (24, 20, 12), (12, 36, 10), (48, 64, 32), (40, 24, 9), (15, 24, 16)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_mixed_form_on_general_grids(monkeypatch, dims, bc):
    """Three steps of the mixed form against the FP64 form, and the interleaved
    viscous solves against one solve after another, bit for bit (FP64 defects in
    both; extents with an odd one keep Jacobi sweeps, one solve after another).
    A viscous solve's velocity error is at most tol |b|, a projection's
    tol |div u| / (2 pi) <= 2 sqrt(3) n / (2 pi) tol |u| = 22 tol |u|: six
    sub-steps of both in two forms, 300 tol |u| in the 2-norm."""
    ref, _ = _steps(dims, bc, capi.FP64)
    got, _ = _steps(dims, bc, capi.MIXED)
    norm = np.sqrt(sum(np.sum(a * a) for a in ref))
    for a, b in zip(ref, got):
        assert np.linalg.norm(a - b) <= 300 * TOL * norm
    monkeypatch.setenv("AFMIB_HELM_DF", "0")
    one, n1 = _steps(dims, bc, capi.MIXED)
    monkeypatch.setenv("AFMIB_HELM_OVERLAP", "0")
    two, n2 = _steps(dims, bc, capi.MIXED)
    assert n1 == n2
    for a, b in zip(one, two):
        assert np.array_equal(a, b)
