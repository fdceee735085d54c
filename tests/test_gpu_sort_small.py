"""The one-block sort and tile ranges (k_sort_small), at the ends of its row counts."""
import numpy as np
import pytest

from afmibins_gb300 import capi

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
SMALL = 16384  # markers up to which one block sorts


@pytest.mark.parametrize("dims", [(24, 16, 32), (64, 64, 64), (40, 24, 1)])
@pytest.mark.parametrize("m", [1, 33, 2048, 2049, 8192, 8193, SMALL])
def test_small_sort_against_passes(dims, m):
    """Spreading of m markers against the same with markers of zero force added
    beyond the one-block sort's range: faces differ by the order of at most m + 64
    terms. Interpolation at the sorted markers bit for bit (a marker's own sum)."""
    n = max(dims)
    rng = np.random.default_rng(m)
    X = rng.uniform(0, np.array(dims) / n, (m + SMALL, 3))
    X[: m // 3] = X[0] + rng.uniform(0, 0.2 / n, (m // 3, 3))  # many of one cell
    if dims[2] == 1:
        X[:, 2] = 0.5 / n
    F = rng.standard_normal((3, m + SMALL))
    F[:, m:] = 0.0
    Fm = F[:, :m].copy()
    N = int(np.prod(dims))
    u, v, w = (rng.standard_normal(N) for _ in range(3))
    with capi.Solver(*dims, n=n, bc=capi.BC_PERIODIC) as sv:
        a = sv.spread(X[:m], Fm)
        b = sv.spread(X, F)
        ia = sv.interp(X[:m], u, v, w)
        ib = sv.interp(X, u, v, w)
    for p, q in zip(a, b):
        assert np.max(np.abs(p - q)) <= (m + 64) * 4 * EPS * max(np.max(np.abs(q)), 1e-300)
    assert np.array_equal(np.asarray(ia), np.asarray(ib)[..., :m])
