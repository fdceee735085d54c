"""Single-operator calls on the caller's device buffers, used in place where they
are memory of the solver's device and no output overlaps another buffer of the
call: the same bits as from host memory, for plain buffers, buffers that start
8 bytes past a 16-byte boundary, the same buffer for several inputs, in-place
calls and partly overlapping outputs."""
import ctypes

import numpy as np
import pytest

from afmibins_gb300 import capi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DIMS = [((16, 12, 20), 0), ((16, 12, 20), 1), ((21, 9, 15), 0), ((16, 12, 1), 0)]


def _dev(a, shift):
    """A device copy of a, `shift` doubles into its allocation."""
    t = torch.zeros(a.size + shift, dtype=torch.float64, device="cuda")
    t[shift:] = torch.from_numpy(np.ascontiguousarray(a).ravel())
    return t[shift:]


def _ops(sv, g):
    """name -> (inputs, output sizes, call(in pointers, out pointers))"""
    N, nv, L, h = sv.ncell, sv.nv, sv.lib, sv.h
    rng = np.random.default_rng(1)
    f = lambda n: rng.standard_normal(n)
    ops = {
        "advection": ([f(N), f(nv), f(N)], [N, nv, N], lambda i, o: L.afmib_advection(h, *o, *i)),
        "div": ([f(N), f(nv), f(N)], [N], lambda i, o: L.afmib_div(h, *o, *i, None, None)),
        "grad": ([f(N)], [N, nv, N], lambda i, o: L.afmib_grad(h, *o, *i)),
        "lap": ([f(N)], [N], lambda i, o: L.afmib_lap_apply(h, *o, *i)),
        "helm0": ([f(N)], [N], lambda i, o: L.afmib_helm_apply(h, 0, -1e-3, *o, *i)),
        "helm1": ([f(nv)], [nv], lambda i, o: L.afmib_helm_apply(h, 1, -1e-3, *o, *i)),
    }
    if all(d % 2 == 0 for d in g[:2]) and (g[2] == 1 or g[2] % 2 == 0):
        nc = N // (4 if g[2] == 1 else 8)
        ops["restrict"] = ([f(N)], [nc], lambda i, o: L.afmib_restrict(h, *o, *i))
        ops["prolong"] = ([f(nc)], [N], lambda i, o: L.afmib_prolong(h, *o, *i))
    if all(d % 4 == 0 for d in g[:2]) and (g[2] == 1 or g[2] % 4 == 0):
        M, n = 50, max(g)
        X = rng.uniform(3.0 / n, (np.array([g[0], g[1], max(g[2], 7)]) - 3.0) / n, (M, 3))
        if g[2] == 1:
            X[:, 2] = 0.5 / n
        ops["spread"] = ([X.ravel(), f(3 * M), rng.uniform(1, 2, M)], [N, nv, N],
                         lambda i, o: L.afmib_spread(h, M, i[0], i[1], i[2], *o))
        ops["interp"] = ([X.ravel(), f(N), f(nv), f(N)], [3 * M], lambda i, o: L.afmib_interp(h, M, *i, *o))
    return ops


@pytest.mark.parametrize("dims,bc", DIMS)
@pytest.mark.parametrize("shift", [0, 1])
def test_device_buffers_match_host(dims, bc, shift):
    with capi.Solver(*dims, n=max(dims), bc=bc) as sv:
        for name, (ins, outs, call) in _ops(sv, dims).items():
            host = [np.full(k, 7.0) for k in outs]
            assert call([capi.ptr(a) for a in ins], [capi.ptr(a) for a in host]) == 0, name
            di = [_dev(a, shift) for a in ins]
            do = [_dev(np.full(k, 7.0), shift) for k in outs]
            torch.cuda.synchronize()
            assert call([capi.ptr(a) for a in di], [capi.ptr(a) for a in do]) == 0, name
            for a, b in zip(host, do):
                assert np.array_equal(a, b.cpu().numpy()), name
            for a, b in zip(ins, di):
                assert np.array_equal(a, b.cpu().numpy()), name  # inputs untouched


@pytest.mark.parametrize("dims,bc", DIMS[:2])
def test_overlapping_device_buffers(dims, bc):
    """In place, one buffer for all inputs, and an output that overlaps an input
    by half, against the host call on copies."""
    with capi.Solver(*dims, n=max(dims), bc=bc) as sv:
        N, nv, L, h, p = sv.ncell, sv.nv, sv.lib, sv.h, capi.ptr
        a = np.random.default_rng(2).standard_normal(2 * N)
        ref = np.zeros(N)
        assert L.afmib_lap_apply(h, p(ref), p(a[:N].copy())) == 0
        t = _dev(a, 0)
        torch.cuda.synchronize()
        assert L.afmib_lap_apply(h, p(t[:N]), p(t[:N])) == 0  # in place
        assert np.array_equal(t[:N].cpu().numpy(), ref)
        t = _dev(a, 0)
        torch.cuda.synchronize()
        assert L.afmib_lap_apply(h, p(t[N // 2:N // 2 + N]), p(t[:N])) == 0  # half an overlap
        assert np.array_equal(t[N // 2:N // 2 + N].cpu().numpy(), ref)
        ins = [a[:N].copy(), a[:nv].copy(), a[:N].copy()]
        refs = [np.zeros(N), np.zeros(nv), np.zeros(N)]
        assert L.afmib_advection(h, *(p(b) for b in refs), *(p(b) for b in ins)) == 0
        t = _dev(a, 0)
        out = [torch.zeros(b.size, dtype=torch.float64, device="cuda") for b in refs]
        torch.cuda.synchronize()
        assert L.afmib_advection(h, *(p(b) for b in out), p(t[:N]), p(t[:nv]), p(t[:N])) == 0
        for b, r in zip(out, refs):
            assert np.array_equal(b.cpu().numpy(), r)
        t = _dev(a, 0)
        torch.cuda.synchronize()
        assert L.afmib_advection(h, p(t[:N]), p(out[1]), p(out[2]), p(t[:N]), p(t[:nv]), p(t[:N])) == 0  # u in place
        assert np.array_equal(t[:N].cpu().numpy(), refs[0]) and np.array_equal(out[2].cpu().numpy(), refs[2])


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("comp,bc", [(0, 0), (1, 0), (2, 1), (1, 1)])
def test_helmholtz_cg_device(comp, bc, shift):
    """The solve in place on the caller's x (and right-hand side the same buffer)."""
    dims = (18, 10, 14)
    with capi.Solver(*dims, n=18, bc=bc, tol=1e-11) as sv:
        n = sv.nv if comp == 1 else sv.ncell
        rng = np.random.default_rng(4)
        b, x0 = rng.standard_normal(n), rng.standard_normal(n)
        ref, it = sv.helmholtz_cg(comp, -1e-3, x0, b)
        x, bd, its = _dev(x0, shift), _dev(b, shift), ctypes.c_int(0)
        torch.cuda.synchronize()
        assert sv.lib.afmib_helmholtz_cg(sv.h, comp, -1e-3, capi.ptr(x), capi.ptr(bd), ctypes.byref(its)) == 0
        # 8-byte aligned vectors take the scalar kernels: the same operations, the norms' sums in another order
        assert its.value == it and np.max(np.abs(x.cpu().numpy() - ref)) <= 1e-13 * np.max(np.abs(ref))
        if shift == 0:
            assert np.array_equal(x.cpu().numpy(), ref)
        same, its = sv.helmholtz_cg(comp, -1e-3, b, b)
        t = _dev(b, shift)
        torch.cuda.synchronize()
        assert sv.lib.afmib_helmholtz_cg(sv.h, comp, -1e-3, capi.ptr(t), capi.ptr(t), None) == 0
        assert np.array_equal(t.cpu().numpy(), same)
