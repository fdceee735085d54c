"""The one-pass smoothing sweep from zero, at the edges of its blocks."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

DIMS = [(128, 12, 8), (132, 20, 12), (48, 64, 40), (64, 36, 36), (96, 48, 80)]


@pytest.mark.parametrize("dims", DIMS + [(128, 96, 1)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_multigrid_first_sweep_keeps_bits(monkeypatch, dims, bc, precision):
    """A sweep that forms its reds from b gives the bits of a cleared x and the two
    colours (AFMIB_INIT_SWEEP=0), with and without over-relaxation, one and four
    cells per thread."""
    if dims[2] == 1 and bc == capi.BC_CHANNEL:
        pytest.skip("2D grids are periodic")
    g = po.Grid(*dims, max(dims), channel=bc == capi.BC_CHANNEL)
    b = np.random.default_rng(5).standard_normal(g.ncell)
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("AFMIB_INIT_SWEEP", mode)
        with capi.Solver(*dims, n=max(dims), bc=bc, precision=precision, tol=1e-8) as sv:
            out[mode] = sv.mg_solve(b)
    assert out["0"][1] == out["1"][1] and np.array_equal(out["0"][0], out["1"][0])


@pytest.mark.parametrize("dims", DIMS + [(32, 20, 6)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_viscous_first_sweep(monkeypatch, dims, bc):
    """One FP32 correction per viscous solve (a loose stopping rule, a single
    sweep): the one-pass sweep against the two colours. The sweeps differ in FP32
    roundings (a dozen per cell, products of b and H's coefficients), the step's
    other passes not at all."""
    g = po.Grid(*dims, 64, channel=bc == capi.BC_CHANNEL)
    rng = np.random.default_rng(6)
    u, v, w = (rng.standard_normal(k) for k in (g.ncell, g.nv, g.ncell))
    monkeypatch.setenv("AFMIB_GS_SWEEPS", "1")
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("AFMIB_INIT_SWEEP", mode)
        with capi.Solver(*dims, n=64, bc=bc, precision=capi.MIXED, mu=0.01, dt=1e-3, tol=0.2) as sv:
            sv.set_velocity(u, v, w)
            sv.ns_step(*(np.zeros(k) for k in (g.ncell, g.nv, g.ncell)))
            out[mode] = sv.get_velocity(), sv.stats()["outer_iters"]
    assert out["0"][1] == out["1"][1]
    top = max(np.abs(a).max() for a in out["0"][0])
    for a, b in zip(out["0"][0], out["1"][0]):
        assert np.max(np.abs(a - b)) <= 64 * 2.0 ** -24 * top
