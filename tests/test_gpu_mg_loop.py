"""The FP64 solve loop decided on the device against the host's loop."""
import numpy as np
import pytest

from afmibins_gb300 import capi

pytestmark = pytest.mark.gpu


def _solve(monkeypatch, graphs, dims, b, **kw):
    monkeypatch.setenv("AFMIB_GRAPHS", graphs)
    with capi.Solver(*dims, n=max(dims), bc=capi.BC_PERIODIC, **kw) as sv:
        out = []
        for rhs in b:
            try:
                x, c = sv.mg_solve(rhs)
                out.append((c, x.tobytes()))
            except Exception as e:
                out.append(str(e))
        return out, sv.stats()["mg_cycles"]


@pytest.mark.parametrize("dims", [(32, 32, 32), (48, 40, 1), (40, 24, 56)])
def test_device_loop_equals_host_loop(monkeypatch, dims):
    """Cycles and bits of several solves on one solver, a solve that starts
    converged, one that meets the cycle cap and one that is not finite: the same
    results, errors and counts, and the solver goes on working after each."""
    rng = np.random.default_rng(9)
    n = int(np.prod(dims))
    b, c = rng.standard_normal(n), rng.standard_normal(n)
    bad = b.copy()
    bad[7] = np.nan
    for kw in (dict(tol=1e-9), dict(tol=1e-9, max_mg_cycles=2)):
        rhs = [b, np.zeros(n), c, bad, b]
        host, dev = (_solve(monkeypatch, g, dims, rhs, **kw) for g in ("0", "1"))
        assert host == dev
        assert dev[0][0] == dev[0][4]
        assert isinstance(dev[0][3], str)
        assert isinstance(dev[0][0], str) == ("max_mg_cycles" in kw)
