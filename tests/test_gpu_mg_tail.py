"""The V-cycle tail (kernels_tail.cu: the coarse levels in one thread-block
cluster, the coarsest solved directly) against the level launches and the CPU
oracle, on grids at the edges of its slab split: one plane per CTA, several, a
last CTA with fewer, 2D rows, ragged extents with a coarsest level of hundreds of
cells, and grids that are a single level."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

GRIDS = [(8, 8, 8), (16, 16, 16), (24, 20, 28), (30, 30, 30), (36, 12, 20), (16, 8, 64), (52, 44, 36), (64, 32, 32),
         (4, 4, 1), (16, 16, 1), (48, 40, 1), (128, 128, 1), (128, 256, 1)]


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("dims", GRIDS)
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_tail_equals_level_launches(monkeypatch, bc, dims, precision):
    """Bit for bit the launch-by-launch V-cycle, and the solver's stop on the
    oracle's residual (the tolerance plus the rounding of evaluating it)."""
    if bc == capi.BC_CHANNEL and dims[2] == 1:
        pytest.skip("2D grids are periodic")
    n, tol = max(dims), 1e-8
    g = po.Grid(*dims, n, channel=bc == capi.BC_CHANNEL)
    b = np.random.default_rng(5).standard_normal(g.ncell)
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("AFMIB_MG_TAIL", mode)
        with capi.Solver(*dims, n=n, bc=bc, precision=precision, tol=tol) as sv:
            out[mode] = sv.mg_solve(b)
    assert out["0"][1] == out["1"][1]
    assert np.array_equal(out["0"][0], out["1"][0])
    r = (b - b.mean()) - po.lap_apply(g, out["1"][0])
    assert np.sqrt(np.mean(r * r)) <= 1.01 * tol


@pytest.mark.parametrize("dims", [(15, 9, 7), (21, 17, 27), (33, 25, 1)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_single_level_direct_solve(bc, dims):
    """An odd grid has one level: the direct solve is the whole solve. Its error
    is the rounding of six dense transforms of at most 33 terms and of the
    eigenvalues, a few hundred units of 2^-53 of the right-hand side."""
    if bc == capi.BC_CHANNEL and dims[2] == 1:
        pytest.skip("2D grids are periodic")
    n = max(dims)
    g = po.Grid(*dims, n, channel=bc == capi.BC_CHANNEL)
    b = np.random.default_rng(6).standard_normal(g.ncell)
    with capi.Solver(*dims, n=n, bc=bc, tol=1e-10) as sv:
        x, _ = sv.mg_solve(b)
    r = (b - b.mean()) - po.lap_apply(g, x)
    assert np.linalg.norm(r) <= 1e-12 * np.linalg.norm(b)
    assert abs(x.mean()) <= 1e-12 * np.abs(x).max()
