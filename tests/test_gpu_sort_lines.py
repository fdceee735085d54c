"""Where the one-block marker sort gives way to the passes over all SMs."""
import numpy as np
import pytest

from afmibins_gb300 import capi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,m,one_block", [((32, 32, 32), 1, True), ((32, 32, 32), 8192, True),
                                              ((32, 32, 32), 8193, False), ((512, 256, 256), 512, True),
                                              ((512, 256, 264), 512, False)])
def test_one_block_up_to_8192_markers_and_65536_tiles(dims, m, one_block):
    """The sort is one launch on one side of the line and at least four on the other;
    spread forces add up to the markers' (64 m products of weights that add up to one,
    each within a few roundings, and a sum over the cells)."""
    n = max(dims)
    N = int(np.prod(dims))
    rng = np.random.default_rng(m)
    X = torch.from_numpy(rng.uniform(0, 1, (m, 3)) * np.array(dims) / n).cuda()
    F = torch.from_numpy(rng.uniform(1, 2, (3, m))).cuda()
    f = [torch.empty(N, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    with capi.Solver(*dims, n=n, bc=capi.BC_PERIODIC) as sv:
        before = sv.stats()["kernel_launches"]
        assert sv.lib.afmib_spread(sv.h, m, capi.ptr(X), capi.ptr(F), None, *(capi.ptr(a) for a in f)) == 0
        launches = sv.stats()["kernel_launches"] - before - 3  # weights, tiles, spreading
    assert launches == 1 if one_block else launches >= 4
    for a, g in zip(f, F):
        assert abs(float(a.sum()) / n ** 3 - float(g.sum())) <= 1e-13 * float(g.sum())
