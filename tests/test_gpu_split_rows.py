"""The FP32 fine level split by colour within its rows against interleaved rows."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(256, 32, 16), (256, 16, 4), (512, 32, 8), (256, 64, 256)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_split_fine_level_keeps_bits(monkeypatch, dims, bc):
    """Solves of the mixed form with x and b of the fine level split by colour and
    with AFMIB_SPLIT=0: the layout changes no arithmetic, so the same bits and
    cycles, over several solves of one solver."""
    g = po.Grid(*dims, 256, channel=bc == capi.BC_CHANNEL)
    rng = np.random.default_rng(14)
    rhs = [rng.standard_normal(g.ncell) for _ in range(2)]
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("AFMIB_SPLIT", mode)
        with capi.Solver(*dims, n=256, bc=bc, precision=capi.MIXED, tol=1e-7) as sv:
            out[mode] = [sv.mg_solve(b) for b in rhs]
    for (x0, c0), (x1, c1) in zip(out["0"], out["1"]):
        assert c0 == c1 and np.array_equal(x0, x1)
