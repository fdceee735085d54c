"""The tile spreading (k_spread_tiles) against the oracle where its staging and
shares can go wrong: markers on both sides of a chunk, chunks that end inside a
plane's range, tiles of 4 and 8 cells, grids two tiles wide (a tile's left and
right neighbour are the same one), channel walls, 2D, volumes, and all markers in
one cell or one plane."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

# 64 contributions a face at most per marker, summed in FP64 in another order than
# the oracle's: rounding of m terms, relative to the largest face
EPS = 2.0 ** -53


@pytest.mark.parametrize("dims,bc", [((16, 16, 16), 0), ((12, 20, 8), 0), ((24, 16, 32), 0), ((16, 24, 16), 1),
                                     ((12, 12, 12), 1), ((16, 24, 1), 0), ((12, 20, 1), 0)])
@pytest.mark.parametrize("m,shape", [(1, "box"), (191, "box"), (193, "plane"), (700, "cell"), (2500, "box")])
def test_spread_tiles_against_oracle(dims, bc, m, shape):
    n = max(dims)
    g = po.Grid(*dims, n, channel=bc == 1)
    rng = np.random.default_rng(3)
    hi = np.array(dims) / n
    lo = np.zeros(3)
    if bc == 1:
        lo[1], hi[1] = 2.6 / n, hi[1] - 2.6 / n
    X = rng.uniform(lo, hi, (m, 3))
    if shape == "plane":  # one plane of cells: a single warp's range without equal shares
        X[:, 2] = (dims[2] // 2 + 0.3) / n
    if shape == "cell":
        X = (np.array(dims) // 2 + rng.uniform(0, 1, (m, 3))) / n
    if dims[2] == 1:
        X[:, 2] = 0.5 / n
    F = rng.standard_normal((3, m))
    vol = rng.uniform(0.5, 2.0, m)
    with capi.Solver(*dims, n=n, bc=bc) as sv:
        out = sv.spread(X, F, vol)
        again = sv.spread(X, F, vol)
        plain = sv.spread(X, F)
    for c in range(3):
        for f, v in ((out, vol), (plain, None)):
            ref = po.spread(g, c, X, F[c].copy(), v)
            assert np.max(np.abs(f[c] - ref)) <= (m + 64) * 4 * EPS * max(np.max(np.abs(ref)), 1e-300)
        assert np.array_equal(out[c], again[c])
