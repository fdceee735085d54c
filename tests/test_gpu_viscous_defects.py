"""The mixed form's viscous solves off the power-of-two extents: FP64 defects."""
import numpy as np
import pytest

from afmibins_gb300 import capi
from oracle import pyoracle as po

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _both(monkeypatch, run):
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("AFMIB_HELM_DF", mode)
        out[mode] = run()
    for a, b in zip(out["0"], out["1"]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dims", [(40, 24, 16), (12, 36, 10), (64, 32, 4)])
@pytest.mark.parametrize("bc", [capi.BC_PERIODIC, capi.BC_CHANNEL])
def test_steps_take_fp64_defects(monkeypatch, dims, bc):
    """AFMIB_HELM_DF=0 asks for an FP64 defect after every correction: on these
    extents (and a power-of-two grid of fewer than eight planes) the default takes
    them too, so both give the same bits."""
    n = max(dims)
    g = po.Grid(*dims, n, channel=bc == capi.BC_CHANNEL)
    rng = np.random.default_rng(41)
    vel = [0.1 * rng.standard_normal(k) for k in (g.ncell, g.nv, g.ncell)]
    f = [rng.standard_normal(k) for k in (g.ncell, g.nv, g.ncell)]

    def run():
        with capi.Solver(*dims, n=n, bc=bc, precision=capi.MIXED, mu=0.01, rho=1.0, dt=1e-3, tol=1e-10) as sv:
            sv.set_velocity(*vel)
            sv.project()
            for _ in range(4):
                sv.ns_step(*f)
            return sv.get_velocity()

    _both(monkeypatch, run)


def test_gradient_takes_fp64_defects(monkeypatch):
    """The same for the reverse pass's solves."""
    from afmibins_gb300.autograd import ib_trajectory, membrane_loss
    dims = (48, 40, 32)
    rng = np.random.default_rng(42)
    X, nstart, nidx = _shell(200)
    v0 = [torch.from_numpy(0.1 * rng.standard_normal(int(np.prod(dims)))).cuda() for _ in range(3)]

    def run():
        with capi.Solver(*dims, n=48, bc=capi.BC_PERIODIC, precision=capi.MIXED, mu=0.01, rho=1.0, dt=1e-4, tol=1e-11,
                         k_spring=0.5) as sv:
            sv.set_velocity(*v0)
            sv.project()
            sv.set_markers(X, nstart, nidx)
            start = [torch.empty_like(a) for a in v0]
            sv.get_velocity(start)
            k = torch.tensor(0.5, dtype=torch.float64, device="cuda", requires_grad=True)
            X0 = torch.from_numpy(X).cuda().requires_grad_(True)
            uN, XN = ib_trajectory(k, X0, sv, tuple(start), 2, 1)
            membrane_loss(uN, XN, X0.detach(), 1.0 / 48 ** 3).backward()
            return [t.detach().cpu().numpy() for t in (uN, XN, k.grad, X0.grad)]

    _both(monkeypatch, run)


def _shell(m):
    """A ring of m markers, each sprung to its two neighbours."""
    t = 2 * np.pi * np.arange(m) / m
    X = np.stack([0.5 + 0.2 * np.cos(t), 0.4 + 0.2 * np.sin(t), np.full(m, 0.3)], 1)
    a = np.arange(m, dtype=np.int32)
    nidx = np.stack([(a - 1) % m, (a + 1) % m], 1).astype(np.int32).ravel()
    return X, (2 * np.arange(m + 1)).astype(np.int32), nidx
