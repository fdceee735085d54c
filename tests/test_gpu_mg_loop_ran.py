"""The FP64 solve loop on the device runs there, instead of falling back unseen to the
host's loop, whose results are the same."""
import numpy as np
import pytest

from afmibins_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 32, 32), (48, 40, 1), (40, 24, 56)])
def test_device_loop_ran(monkeypatch, dims):
    """One more kernel than the host's loop per V-cycle and one before the first: the
    one-thread test of the residual."""
    b = np.random.default_rng(3).standard_normal(int(np.prod(dims)))
    launches = {}
    for graphs in ("0", "1"):
        monkeypatch.setenv("AFMIB_GRAPHS", graphs)
        with capi.Solver(*dims, n=max(dims), bc=capi.BC_PERIODIC, tol=1e-9) as sv:
            _, cycles = sv.mg_solve(b)
            launches[graphs] = sv.stats()["kernel_launches"]
    assert launches["1"] - launches["0"] == cycles + 1
