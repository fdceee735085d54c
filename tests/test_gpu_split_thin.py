"""The FP32 fine level split by colour on its thinnest grids, four planes: one batch
of planes per thread wraps onto itself."""
import numpy as np
import pytest

from afmibins_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(256, 64, 4), (512, 32, 4), (256, 128, 8)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_split_thin_grids_keep_bits(monkeypatch, dims, bc):
    """Above the 32768 cells that the coarse levels' single launch takes, so that the
    fine level has launches of its own: the same bits and cycles with and without the
    split. That it is on shows in the fused residual-restriction, which split rows
    take even where it is switched off."""
    assert int(np.prod(dims)) > 32768
    rng = np.random.default_rng(15)
    rhs = [rng.standard_normal(int(np.prod(dims))) for _ in range(2)]
    out, fused = {}, {}
    for mode in ("0", "1"):
        monkeypatch.setenv("AFMIB_SPLIT", mode)
        monkeypatch.delenv("AFMIB_RESID_RESTRICT", raising=False)
        with capi.Solver(*dims, n=256, bc=bc, precision=capi.MIXED, tol=1e-7) as sv:
            out[mode] = [sv.mg_solve(b) for b in rhs]
            monkeypatch.setenv("AFMIB_RESID_RESTRICT", "0")
            sv.profile(True)
            sv.profile_reset()
            sv.mg_solve(rhs[0])
            fused[mode] = "mg_resid_restrict_fine" in sv.profile_table()
    assert fused == {"0": False, "1": True}
    for (x0, c0), (x1, c1) in zip(out["0"], out["1"]):
        assert c0 == c1 and np.array_equal(x0, x1)
