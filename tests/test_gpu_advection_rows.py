"""The FP64 advection kernel that walks row pairs along z, at the edges of its blocks."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 6, 4), (33, 7, 9), (130, 5, 3), (256, 3, 5), (300, 4, 6), (512, 2, 3), (514, 3, 4)])
@pytest.mark.parametrize("bc", [0, 1])
def test_advection_rows(dims, bc):
    """FP64 advection by row pairs (k_advect_rows: rows of x in one block, chunks
    of planes, an odd last row) against the oracle; the last grid's rows are too
    long for it. The fluxes are products of two sums, differences of six of them:
    a few roundings of n |u|^2."""
    n = max(dims)
    g = po.Grid(*dims, n, channel=bc == 1)
    rng = np.random.default_rng(8)
    u, v, w = rng.standard_normal(g.ncell), rng.standard_normal(g.nv), rng.standard_normal(g.ncell)
    with capi.Solver(*dims, n=n, bc=bc) as sv:
        got = sv.advection(u, v, w)
    top = max(np.abs(a).max() for a in (u, v, w))
    for a, b in zip(got, po.advection(g, u, v, w)):
        assert np.max(np.abs(a - b)) <= 32 * 2.0 ** -53 * n * top ** 2
