"""The V-cycle tail on smaller clusters than the device's largest: other slabs, other
levels behind it, and levels with more cells than a CTA's threads take at once."""
import numpy as np
import pytest

from afmibins_gb300 import capi

pytestmark = pytest.mark.gpu

GRIDS = [(16, 16, 16), (24, 20, 28), (30, 30, 30), (32, 32, 32), (16, 8, 64), (64, 64, 8), (64, 32, 16), (52, 44, 36),
         (48, 40, 1), (128, 128, 1), (128, 256, 1)]


def _solve(monkeypatch, dims, bc, precision, b, **env):
    for k in ("AFMIB_MG_TAIL", "AFMIB_MG_TAIL_CLUSTER"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with capi.Solver(*dims, n=max(dims), bc=bc, precision=precision, tol=1e-8) as sv:
        return sv.mg_solve(b)


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("dims", GRIDS)
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_every_cluster_equals_level_launches(monkeypatch, bc, dims, precision):
    """Bit for bit the launch-by-launch V-cycle on 16, 8, 4, 2 and 1 CTAs."""
    if bc == capi.BC_CHANNEL and dims[2] == 1:
        pytest.skip("2D grids are periodic")
    b = np.random.default_rng(7).standard_normal(int(np.prod(dims)))
    x0, c0 = _solve(monkeypatch, dims, bc, precision, b, AFMIB_MG_TAIL="0")
    for cluster in ("16", "8", "4", "2", "1"):
        x, c = _solve(monkeypatch, dims, bc, precision, b, AFMIB_MG_TAIL_CLUSTER=cluster)
        assert c == c0 and np.array_equal(x, x0), cluster


@pytest.mark.parametrize("dims,clusters", [((15, 9, 7), "8421"), ((21, 17, 27), "842"), ((33, 25, 1), "8421")])
def test_direct_solve_on_smaller_clusters(monkeypatch, dims, clusters):
    """The coarsest level's transforms: each plane's sums have the same terms in the
    same order wherever the plane lies (21 x 17 x 27 cells do not fit one CTA)."""
    b = np.random.default_rng(8).standard_normal(int(np.prod(dims)))
    ref = _solve(monkeypatch, dims, capi.BC_PERIODIC, capi.FP64, b)
    for cluster in clusters:
        got = _solve(monkeypatch, dims, capi.BC_PERIODIC, capi.FP64, b, AFMIB_MG_TAIL_CLUSTER=cluster)
        assert got[1] == ref[1] and np.array_equal(got[0], ref[0]), cluster
