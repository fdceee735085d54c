"""The work a user of this framework has it do, as measurable cases.

Every case is one pass through the public entry points: whole immersed-boundary
steps in both precisions, a channel flow step, the gradient of a short run, a
projection, a viscous solve, the marker transfers and single MAC operators on
the caller's device buffers. `listed()` holds one case of each kind of use from
the smallest call to the largest grid, `draw(rng)` more of the same ranges,
`exact(case, seed)` the same outputs in 64 bits from plain torch (spectral
solves in the periodic directions, an eigenbasis in y between walls).

Fields are flat FP64 arrays, x fastest; the face convention is the package's:
u at (x, y+1/2, z+1/2), v at (x+1/2, y, z+1/2), w at (x+1/2, y+1/2, z), and v
holds the ny-1 interior planes between channel walls.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from afmibins_gb300 import capi
from afmibins_gb300 import markers as mk
from afmibins_gb300.autograd import ib_trajectory, membrane_loss

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # production forward run in the mixed form: many shells in a turbulent box
        dict(name="ib_mixed_256", kind="ib", nx=256, ny=256, nz=256, precision="mixed", shells=10, per_shell=20000,
             radius=0.08, mu=0.005, dt=2e-5, k=0.5, kb=0.0, tol=1e-10),
        # the largest run one GPU takes in earnest: 512^3 with a million markers
        dict(name="ib_mixed_512", kind="ib", nx=512, ny=512, nz=512, precision="mixed", shells=40, per_shell=25000,
             radius=0.05, mu=0.002, dt=1e-5, k=0.5, kb=0.0, tol=1e-10),
        # the FP64 drop-in on one spherical shell
        dict(name="ib_fp64_128", kind="ib", nx=128, ny=128, nz=128, precision="fp64", shells=1, per_shell=20480,
             radius=0.2, mu=0.01, dt=5e-5, k=0.5, kb=0.0, tol=1e-10),
        # the small two-dimensional run: one closed membrane, launch latency
        dict(name="ib_fp64_2d_128", kind="ib", nx=128, ny=128, nz=1, precision="fp64", shells=1, per_shell=512,
             radius=0.25, mu=0.01, dt=1e-4, k=1.0, kb=0.0, tol=1e-12),
        # a box that is no cube and no power of two, with bending membranes
        dict(name="ib_mixed_box", kind="ib", nx=96, ny=80, nz=112, precision="mixed", shells=3, per_shell=2500,
             radius=0.15, mu=0.01, dt=1e-4, k=0.5, kb=1e-3, tol=1e-10),
        # channel flow between moving walls with a body force, one full step (BE and CN sub-steps)
        dict(name="ns_channel_96", kind="ns", nx=96, ny=64, nz=64, channel=True, precision="fp64", corrected=0,
             mu=0.01, dt=2e-4, tol=1e-10),
        # a divergence-free start field: one projection on its own
        dict(name="project_mixed_128", kind="project", nx=128, ny=128, nz=128, channel=False, precision="mixed",
             tol=1e-10),
        # one implicit viscous solve on a ragged grid, as a caller with its own time stepping asks for it
        dict(name="helmholtz_120", kind="helmholtz", nx=120, ny=90, nz=70, channel=False, comp=0, off=0.25, tol=1e-10),
        # a caller with its own fluid solver: spread marker forces, interpolate velocities
        dict(name="transfers_256", kind="transfers", nx=256, ny=256, nz=256, channel=False, shells=10,
             per_shell=20000, radius=0.08),
        # the momentum transport of given velocities
        dict(name="advection_192", kind="operator", op="advection", nx=192, ny=160, nz=128, channel=False),
        # the smallest call: one Laplacian on a small grid
        dict(name="laplacian_32", kind="operator", op="laplacian", nx=32, ny=32, nz=32, channel=False),
        # stiffness and shape gradient of a short run through autograd
        dict(name="gradient_64", kind="gradient", nx=64, ny=64, nz=64, precision="mixed", shells=1, per_shell=5120,
             radius=0.2, mu=0.01, dt=1e-4, k=0.5, tol=1e-11, steps=2, every=1),
    ]


def _extent(rng, lo, hi, step=0):
    """An extent log-uniform in [lo, hi]; a multiple of 4, 8 or 16 (the larger the coarser) unless step is given."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    q = step or (4 if n < 48 else 8 if n < 112 else 16)
    return max(lo, min(hi, q * round(n / q)))


def _box(rng, lo, hi, cells, step=0):
    """Extents within a factor of two of each other, at most `cells` cells; powers of two (the grids that coarsen
    furthest) more often than chance."""
    two = not step and rng.random() < 0.4

    def extent(lo, hi):
        n = _extent(rng, lo, hi, step)
        return max(lo, min(hi, 1 << round(math.log2(n)))) if two else n

    while True:
        a = extent(lo, hi)
        e = [a if rng.random() < 0.4 else extent(max(lo, a // 2), min(hi, 2 * a)) for _ in range(2)] + [a]
        rng.shuffle(e)
        if e[0] * e[1] * e[2] <= cells:
            return dict(nx=e[0], ny=e[1], nz=e[2])


def _membranes(rng, g):
    """Shells of about three markers per squared cell that fit the box."""
    n = max(g["nx"], g["ny"], g["nz"])
    side = min(g["nx"], g["ny"], g["nz"]) / n
    shells = rng.choice([1, 1, 2, 4, 8])
    radius = side * (rng.uniform(0.15, 0.25) if shells < 3 else rng.uniform(0.07, 0.11))
    per = int(rng.uniform(2.0, 4.0) * 4 * math.pi * (radius * n) ** 2)
    return dict(shells=shells, per_shell=max(64, per), radius=round(radius, 4))


def draw(rng):
    kind = rng.choice(["ib", "ib", "ib2d", "ns", "project", "helmholtz", "transfers", "operator", "operator",
                       "gradient"])
    if kind == "ib":
        mixed = rng.random() < 0.6
        g = _box(rng, 32, 256, 256 ** 3 if mixed else 128 ** 3)
        n = max(g["nx"], g["ny"], g["nz"])
        return dict(kind="ib", **g, precision="mixed" if mixed else "fp64", **_membranes(rng, g),
                    mu=rng.choice([0.005, 0.01]), dt=round(rng.uniform(4e-3, 8e-3) / n, 8), k=0.5,
                    kb=rng.choice([0.0, 0.0, 1e-3]), tol=1e-10)
    if kind == "ib2d":
        a = _extent(rng, 64, 512)
        b = a if rng.random() < 0.5 else _extent(rng, max(64, a // 2), min(512, 2 * a))
        n = max(a, b)
        return dict(kind="ib", nx=a, ny=b, nz=1, precision=rng.choice(["fp64", "mixed"]), shells=1,
                    per_shell=int(4 * n * rng.uniform(0.8, 1.2)), radius=round(0.25 * min(a, b) / n, 4), mu=0.01,
                    dt=round(0.0128 / n, 8), k=1.0, kb=0.0, tol=1e-10)
    if kind == "ns":
        mixed = rng.random() < 0.5
        g = _box(rng, 32, 192, 192 ** 3 if mixed else 112 ** 3)
        n = max(g["nx"], g["ny"], g["nz"])
        channel = rng.random() < 0.7
        return dict(kind="ns", **g, channel=channel, precision="mixed" if mixed else "fp64",
                    corrected=rng.choice([0, 1]) if g["ny"] <= g["nz"] else 1, mu=0.01, dt=round(0.0128 / n, 8),
                    tol=1e-10)
    if kind == "project":
        mixed = rng.random() < 0.5
        return dict(kind="project", **_box(rng, 32, 256, 256 ** 3 if mixed else 128 ** 3), channel=rng.random() < 0.4,
                    precision="mixed" if mixed else "fp64", tol=1e-10)
    if kind == "helmholtz":
        channel = rng.random() < 0.4
        return dict(kind="helmholtz", **_box(rng, 20, 200, 160 ** 3, 2), channel=channel, comp=rng.choice([0, 1, 2]),
                    off=round(math.exp(rng.uniform(math.log(0.004), math.log(1.0))), 4), tol=1e-10)
    if kind == "transfers":
        g = _box(rng, 32, 256, 256 ** 3)
        return dict(kind="transfers", **g, channel=rng.random() < 0.4, **_membranes(rng, g))
    if kind == "operator":
        return dict(kind="operator", op=rng.choice(["advection", "laplacian", "helmholtz", "divergence", "gradient"]),
                    **_box(rng, 20, 300, 256 ** 3, 1), channel=rng.random() < 0.4)
    g = _box(rng, 32, 64, 64 ** 3, 8)
    return dict(kind="gradient", **g, precision=rng.choice(["fp64", "mixed"]), **_membranes(rng, g), mu=0.01,
                dt=round(0.0064 / 64, 8), k=0.5, tol=1e-11, steps=2, every=rng.choice([1, 2]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _n(case):
    return max(case["nx"], case["ny"], case["nz"])


def _cells(case):
    return case["nx"] * case["ny"] * case["nz"]


def _channel(case):
    return bool(case.get("channel", False))


def _interior(case, f):
    """The ny-1 interior planes of a v field [nz, ny, nx] between walls."""
    return f[:, 1:, :].contiguous() if _channel(case) else f


def _random_velocity(case, seed, rms=0.1, solenoidal=True):
    """Smooth random field with energy peaked at |k| = 4; its divergence-free part if asked."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 3 + 1)
    kx = torch.fft.rfftfreq(nx, 1.0 / nx, device=DEV, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, 1.0 / ny, device=DEV, dtype=torch.float64)[:, None]
    kz = torch.fft.fftfreq(nz, 1.0 / nz, device=DEV, dtype=torch.float64)[:, None, None]
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    amp = torch.sqrt(k2) * torch.exp(-k2 / 16.0)
    comps = 2 if nz == 1 else 3
    h = [amp * torch.fft.rfftn(torch.randn((nz, ny, nx), dtype=torch.float64, device=DEV, generator=gen))
         for _ in range(comps)]
    if solenoidal:
        kv = [kx, ky, kz][:comps]
        dot = sum(a * b for a, b in zip(h, kv)) / torch.clamp(k2, min=1.0)
        h = [a - b * dot for a, b in zip(h, kv)]
    f = [torch.fft.irfftn(a, s=(nz, ny, nx)) for a in h]
    r = math.sqrt(sum(float((a * a).mean()) for a in f) / len(f))
    f = [a * (rms / r) for a in f]
    if nz == 1:
        f.append(torch.zeros_like(f[0]))
    if _channel(case):
        f[1][:, 0, :] = 0.0
    return f


def _shell_springs(m):
    """Unit-sphere Fibonacci lattice and its symmetric springs: the three lattice directions nearest at the equator."""
    i = np.arange(m) + 0.5
    th = np.arccos(1 - 2 * i / m)
    golden = (1 + 5 ** 0.5) / 2
    ph = 2 * np.pi * i * golden
    P = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1)
    fib = [1, 2]
    while fib[-1] < m:
        fib.append(fib[-1] + fib[-2])
    step = [math.hypot(2 * f / m, 2 * math.pi * abs(f * golden - round(f * golden))) for f in fib]
    offs = sorted(f for _, f in sorted(zip(step, fib))[:3])
    offs = np.array([-f for f in reversed(offs)] + offs)
    j = np.arange(m)[:, None] + offs[None, :]
    keep = (j >= 0) & (j < m)
    return P, keep.sum(1), j, keep


def _membrane(case, seed):
    """Marker positions (device) and neighbour lists (host) of the case's membranes."""
    n, M = _n(case), case["per_shell"]
    rng = np.random.default_rng(int(seed))
    side = [case["nx"] / n, case["ny"] / n, case["nz"] / n]
    if case["nz"] == 1:
        t = 2 * np.pi * np.arange(M) / M + rng.uniform(0, 2 * np.pi / M)
        amp = 0.01 * rng.standard_normal(2)
        r = case["radius"] * (1 + amp[0] * np.cos(2 * t) + amp[1] * np.sin(3 * t))
        X = np.stack([side[0] / 2 + r * np.cos(t), side[1] / 2 + 0.8 * r * np.sin(t), np.full(M, 0.5 / n)], 1)
        a = np.arange(M, dtype=np.int32)
        nidx = np.stack([(a - 1) % M, (a + 1) % M], 1).astype(np.int32).ravel()
        return X, (2 * np.arange(M + 1)).astype(np.int32), nidx
    P, count, j, keep = _shell_springs(M)
    S, r0 = case["shells"], case["radius"]
    lo = [1.3 * r0 + 3.5 / n if _channel(case) and a == 1 else r0 for a in range(3)]
    hi = [max(l + 1e-3, s - l) for s, l in zip(side, lo)]
    gap = 2.2 * r0
    c = []
    while len(c) < S:  # shells apart from one another while there is room
        q = rng.uniform(lo, hi)
        if all(np.linalg.norm(q - o) >= gap for o in c):
            c.append(q)
        else:
            gap *= 0.995
    Xs = []
    for q in c:
        amp = 0.03 * rng.standard_normal()
        Xs.append(q + r0 * (1 + amp * mk.y2(int(rng.integers(-2, 3)), P))[:, None] * P)
    X = np.concatenate(Xs)
    counts = np.tile(count, S)
    nstart = np.zeros(S * M + 1, dtype=np.int32)
    np.cumsum(counts, out=nstart[1:])
    base = j[keep].astype(np.int32)
    nidx = (base[None, :] + (M * np.arange(S, dtype=np.int32))[:, None]).ravel().astype(np.int32)
    return X, nstart, nidx


def _solver(case, **kw):
    prec = capi.MIXED if case.get("precision") == "mixed" else capi.FP64
    return capi.Solver(case["nx"], case["ny"], case["nz"], n=_n(case),
                       bc=capi.BC_CHANNEL if _channel(case) else capi.BC_PERIODIC, precision=prec,
                       tol=case.get("tol", 1e-10), **kw)


def _scale(case):
    """The viscous operator's (I + s Laplacian) scale of a standalone solve."""
    return -case["off"] / float(_n(case)) ** 2


def _forces(case, seed):
    """A body force: a steady streamwise drive and a smooth random part."""
    f = _random_velocity(case, seed + 7, rms=1.0, solenoidal=False)
    f[0] = f[0] + 2.0
    f[1] = _interior(case, f[1])
    return [a.contiguous().reshape(-1) for a in f]


def _walls(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 5 + 2)
    return [0.05 * torch.randn(case["nx"] * case["nz"], dtype=torch.float64, device=DEV, generator=gen)
            for _ in range(4)]


def _marker_forces(case, X, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7 + 3)
    return torch.randn((3, X.shape[0]), dtype=torch.float64, device=DEV, generator=gen)


def _flat(case, f):
    f = list(f)
    f[1] = _interior(case, f[1])
    return [a.contiguous().reshape(-1) for a in f]


def _viscous_inputs(case, seed):
    """Warm start and right-hand side of one component's viscous solve."""
    old = _random_velocity(case, seed)[case["comp"]]
    src = _random_velocity(case, seed + 1, rms=0.02, solenoidal=False)[case["comp"]]
    if case["comp"] == 1:
        old, src = _interior(case, old), _interior(case, src)
    return old.contiguous().reshape(-1), (old + src).contiguous().reshape(-1)


def _provisional(case, seed):
    """A velocity as a projection meets it: mostly divergence-free, with a compressive part."""
    a = _random_velocity(case, seed)
    b = _random_velocity(case, seed + 1, rms=0.01, solenoidal=False)
    return [p + q for p, q in zip(a, b)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    N = _cells(case)
    if kind in ("ib", "gradient"):
        X, nstart, nidx = _membrane(case, seed)
        sv = _solver(case, mu=case["mu"], rho=1.0, dt=case["dt"], k_spring=case["k"], k_bend=case.get("kb", 0.0))
        vel = _flat(case, _random_velocity(case, seed))
        Xd = torch.from_numpy(X).to(DEV)
        torch.cuda.synchronize()
        sv.set_velocity(*vel)
        sv.project()
        sv.set_markers(Xd, nstart, nidx)
        s["sv"] = sv
        if kind == "ib":
            s["vel"] = [torch.empty(N, dtype=torch.float64, device=DEV) for _ in range(3)]
            s["X"] = torch.empty_like(Xd)
        else:
            sv.get_velocity(vel)
            s["vel0"], s["X0"] = tuple(vel), Xd
    elif kind == "ns":
        sv = _solver(case, mu=case["mu"], rho=1.0, dt=case["dt"], walls_corrected=case["corrected"])
        vel = _flat(case, _random_velocity(case, seed))
        s["f"] = _forces(case, seed)
        s["walls"] = _walls(case, seed) if _channel(case) else None
        torch.cuda.synchronize()
        sv.set_velocity(*vel)
        sv.project()
        s["sv"], s["vel"] = sv, [torch.empty_like(a) for a in vel]
    elif kind == "project":
        s["sv"] = _solver(case)
        s["in"] = _flat(case, _provisional(case, seed))
        s["vel"] = [torch.empty_like(a) for a in s["in"]]
    elif kind == "helmholtz":
        s["sv"] = _solver(case)
        s["x0"], s["b"] = _viscous_inputs(case, seed)
        s["x"] = torch.empty_like(s["b"])
    elif kind == "transfers":
        s["sv"] = _solver(case)
        s["X"] = torch.from_numpy(_membrane(case, seed)[0]).to(DEV)
        s["F"] = _marker_forces(case, s["X"], seed)
        s["vel"] = _flat(case, _random_velocity(case, seed))
        s["f"] = [torch.empty_like(a) for a in s["vel"]]
        s["U"] = torch.empty_like(s["F"])
    else:
        s["sv"] = _solver(case)
        s["in"] = _operator_inputs(case, seed)
        s["out"] = [torch.empty(k, dtype=torch.float64, device=DEV) for k in _operator_sizes(case)]
    torch.cuda.synchronize()
    return s


def _operator_inputs(case, seed):
    vel = _flat(case, _random_velocity(case, seed))
    if case["op"] in ("advection", "divergence"):
        return vel
    return [vel[0]]


def _operator_sizes(case):
    N = _cells(case)
    nv = case["nx"] * (case["ny"] - 1) * case["nz"] if _channel(case) else N
    return [N, nv, N] if case["op"] in ("advection", "gradient") else [N]


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ok(sv, status):
    if status != capi.AFMIB_OK:
        raise capi.AfmibError(status, sv.last_error())


def run(state):
    case, sv = state["case"], state["sv"]
    kind, p, L, h = case["kind"], capi.ptr, sv.lib, sv.h
    if kind == "ib":
        sv.ib_step(1)
        sv.get_velocity(state["vel"])
        sv.get_markers(state["X"])
        return state["vel"] + [state["X"]]
    if kind == "gradient":
        k = torch.tensor(case["k"], dtype=torch.float64, device=DEV, requires_grad=True)
        X0 = state["X0"].clone().requires_grad_(True)
        uN, XN = ib_trajectory(k, X0, sv, state["vel0"], case["steps"], case["every"])
        membrane_loss(uN, XN, X0.detach(), 1.0 / _n(case) ** 3).backward()
        return [uN.detach(), XN.detach(), k.grad, X0.grad]
    if kind == "ns":
        if state["walls"] is not None:
            sv.set_walls(*state["walls"])
        for _ in range(2):
            sv.ns_step(*state["f"])
        sv.get_velocity(state["vel"])
        return state["vel"]
    if kind == "project":
        sv.set_velocity(*state["in"])
        sv.project()
        sv.get_velocity(state["vel"])
        return state["vel"]
    if kind == "helmholtz":
        state["x"].copy_(state["x0"])
        torch.cuda.current_stream().synchronize()  # the solver's stream does not wait for torch's
        it = ctypes.c_int(0)
        _ok(sv, L.afmib_helmholtz_cg(h, case["comp"], _scale(case), p(state["x"]), p(state["b"]), ctypes.byref(it)))
        return [state["x"]]
    if kind == "transfers":
        X, F, f, vel = state["X"], state["F"], state["f"], state["vel"]
        _ok(sv, L.afmib_spread(h, X.shape[0], p(X), p(F), None, *(p(a) for a in f)))
        _ok(sv, L.afmib_interp(h, X.shape[0], p(X), *(p(a) for a in vel), p(state["U"])))
        return f + [state["U"]]
    a, o = [p(t) for t in state["in"]], [p(t) for t in state["out"]]
    if case["op"] == "advection":
        _ok(sv, L.afmib_advection(h, *o, *a))
    elif case["op"] == "laplacian":
        _ok(sv, L.afmib_lap_apply(h, *o, *a))
    elif case["op"] == "helmholtz":
        _ok(sv, L.afmib_helm_apply(h, 0, -0.1 / float(_n(case)) ** 2, *o, *a))
    elif case["op"] == "divergence":
        _ok(sv, L.afmib_div(h, *o, *a, None, None))
    else:
        _ok(sv, L.afmib_grad(h, *o, *a))
    return state["out"]


def work(case):
    """Bytes and FP64-equivalent operations no implementation of the pass can do without."""
    N, kind = _cells(case), case["kind"]
    M = case.get("shells", 0) * case.get("per_shell", 0)
    transfer = M * 3 * (64 * 3 + 36)  # one direction, three components, with the weights
    project = N * (8 + 60 + 9)        # divergence, one multigrid cycle's worth of solve, gradient
    substep = N * (66 + 3 * (5 + 2 * 10)) + project
    if kind == "ib":
        return {"bytes": 6 * N * 8 + M * (24 + 24 + 6 * 4), "flops": 2 * substep + 4 * transfer}
    if kind == "gradient":
        return {"bytes": case["steps"] * (12 * N * 8 + M * 96), "flops": case["steps"] * 2.5 * (2 * substep + 4 * transfer)}
    if kind == "ns":
        return {"bytes": 9 * N * 8, "flops": 2 * substep}
    if kind == "project":
        return {"bytes": 6 * N * 8, "flops": project}
    if kind == "helmholtz":
        return {"bytes": 3 * N * 8, "flops": 40 * N}
    if kind == "transfers":
        return {"bytes": 6 * N * 8 + M * (2 * 24 + 48), "flops": 2 * transfer}
    ins = 3 if case["op"] in ("advection", "divergence") else 1
    outs = 3 if case["op"] in ("advection", "gradient") else 1
    per = {"advection": 66, "laplacian": 8, "helmholtz": 9, "divergence": 7, "gradient": 6}[case["op"]]
    return {"bytes": (ins + outs) * N * 8, "flops": per * N}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _xm(f): return torch.roll(f, 1, 2)
def _xp(f): return torch.roll(f, -1, 2)
def _ym(f): return torch.roll(f, 1, 1)
def _yp(f): return torch.roll(f, -1, 1)
def _zm(f): return torch.roll(f, 1, 0)
def _zp(f): return torch.roll(f, -1, 0)


class _Exact:
    """The discrete operators of one case on [nz, ny, nx] tensors (v with its zero wall plane in channel mode)."""

    def __init__(self, case):
        self.case, self.n, self.ch = case, float(_n(case)), _channel(case)
        self.nx, self.ny, self.nz = case["nx"], case["ny"], case["nz"]
        t = lambda m: 2.0 * torch.cos(2 * math.pi * torch.arange(m, dtype=torch.float64, device=DEV) / m) - 2.0
        self.lx, self.ly, self.lz = t(self.nx)[: self.nx // 2 + 1], t(self.ny)[:, None], t(self.nz)[:, None, None]
        if self.ch:
            self.y = {"p": self._ybasis("p"), "u": self._ybasis("u"), "v": self._ybasis("v")}

    def full(self, flat):
        """[nz, ny, nx] from a flat array; v's interior planes get their wall plane."""
        if self.ch and flat.numel() == self.nx * (self.ny - 1) * self.nz:
            f = torch.zeros((self.nz, self.ny, self.nx), dtype=torch.float64, device=DEV)
            f[:, 1:, :] = flat.reshape(self.nz, self.ny - 1, self.nx)
            return f
        return flat.reshape(self.nz, self.ny, self.nx)

    def flat(self, f, comp=0):
        return (f[:, 1:, :] if self.ch and comp == 1 else f).reshape(-1)

    def _ymatrix(self, kind):
        """Second difference in y between walls: pressure (Neumann), u and w (one-sided closure), v (interior faces)."""
        m = self.ny - 1 if kind == "v" else self.ny
        A = np.diag(np.full(m, -2.0)) + np.diag(np.ones(m - 1), 1) + np.diag(np.ones(m - 1), -1)
        if kind == "p":
            A[0, 0] = A[-1, -1] = -1.0
        if kind == "u":
            A[0, 0] = A[-1, -1] = -4.0
            A[0, 1] = A[-1, -2] = 4.0 / 3.0
        return A

    def _ybasis(self, kind):
        A = self._ymatrix(kind)
        D = np.ones(len(A))
        if kind == "u":  # rows 0 and ny-1 scaled so that the matrix is symmetric
            D[0] = D[-1] = math.sqrt(4.0 / 3.0)
        ev, V = np.linalg.eigh(A / D[:, None] * D[None, :])
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
        return to(ev), to(V.T / D[None, :]), to(D[:, None] * V)

    def _solve(self, f, kind, mul):
        """mul(n^2 eigenvalue of the Laplacian) applied in the Laplacian's eigenbasis."""
        n2 = self.n ** 2
        if not self.ch:
            return torch.fft.irfftn(torch.fft.rfftn(f) * mul(n2 * (self.lx + self.ly + self.lz)),
                                    s=(self.nz, self.ny, self.nx))
        ev, fwd, bwd = self.y[kind]
        g = f[:, 1:, :] if kind == "v" else f
        h = torch.fft.rfftn(g, dim=(0, 2))
        h = torch.complex(fwd @ h.real, fwd @ h.imag) * mul(n2 * (self.lx + ev[:, None] + self.lz))
        g = torch.fft.irfftn(torch.complex(bwd @ h.real, bwd @ h.imag), s=(self.nz, self.nx), dim=(0, 2))
        if kind != "v":
            return g
        return torch.cat([torch.zeros_like(f[:, :1, :]), g], 1)

    def lap(self, f, kind="p"):
        n2 = self.n ** 2
        if not self.ch:
            s = _xm(f) + _xp(f) + _ym(f) + _yp(f) - 4.0 * f
            return n2 * (s if self.nz == 1 else s + _zm(f) + _zp(f) - 2.0 * f)
        g = f[:, 1:, :] if kind == "v" else f
        A = torch.from_numpy(self._ymatrix(kind)).to(DEV)
        s = _xm(g) + _xp(g) + _zm(g) + _zp(g) - 4.0 * g + A @ g
        return n2 * (s if kind != "v" else torch.cat([torch.zeros_like(f[:, :1, :]), s], 1))

    def kind(self, comp):
        return "v" if comp == 1 else "u"

    def helm(self, f, s, comp):
        return f + s * self.lap(f, self.kind(comp))

    def helm_solve(self, b, s, comp):
        return self._solve(b, self.kind(comp), lambda l: 1.0 / (1.0 + s * l))

    def wallmask(self, f):
        if not self.ch:
            return f
        m = torch.ones_like(f)
        m[:, 0, :] = 0.0
        return f * m

    def advection(self, u, v, w):
        n = self.n
        uu, vv, ww = ((u + _xm(u)) / 2) ** 2, ((v + _ym(v)) / 2) ** 2, ((w + _zm(w)) / 2) ** 2
        uv = (u + _ym(u)) * (v + _xm(v)) / 4
        uw = (u + _zm(u)) * (w + _xm(w)) / 4
        vw = (v + _zm(v)) * (w + _ym(w)) / 4
        return [n * ((_xp(uu) - uu) + (_yp(uv) - uv) + (_zp(uw) - uw)),
                self.wallmask(n * ((_xp(uv) - uv) + (_yp(vv) - vv) + (_zp(vw) - vw))),
                n * ((_xp(uw) - uw) + (_yp(vw) - vw) + (_zp(ww) - ww))]

    def div(self, u, v, w):
        return self.n * ((_xp(u) - u) + (_yp(v) - v) + (_zp(w) - w))

    def grad(self, p):
        return [self.n * (p - _xm(p)), self.wallmask(self.n * (p - _ym(p))), self.n * (p - _zm(p))]

    def project(self, vel):
        """(projected velocity, gradient)"""
        tiny = 1e-9 * self.n ** 2  # the constant mode
        phi = self._solve(self.div(*vel), "p", lambda l: torch.where(l.abs() < tiny, torch.zeros_like(l), 1.0 / l))
        g = self.grad(phi)
        return [a - b for a, b in zip(vel, g)], g

    def substep(self, old, now, f, half, walls, wallgrad):
        """One sub-step; walls (ut, ub, wt, wb as [nz, nx]) are updated in place. Returns (velocity, gradient)."""
        c = self.case
        dt, n2 = c["dt"], self.n ** 2
        sp, sm = c["mu"] * dt / 2, -c["mu"] * dt / 2
        if walls is not None:
            gx, gz = wallgrad[0], wallgrad[2]
            keep = torch.ones(self.nx * self.nz, dtype=torch.float64, device=DEV)
            gz2 = gz if c["corrected"] else gx
            if not c["corrected"]:
                keep[self.nx * min(self.ny, self.nz):] = 0.0
            keep = keep.reshape(self.nz, self.nx)
            for k, (first, second, e0, e1) in enumerate(((gx, gx, -1, -2), (gx, gx, 0, 1), (gz, gz2, -1, -2), (gz, gz2, 0, 1))):
                walls[k] = walls[k] + keep * (9 * first[:, e0, :] - second[:, e1, :]) / 8
        adv = self.advection(*now)
        new = []
        for comp in range(3):
            src = (dt / 2 if not half else dt) * (f[comp] - adv[comp])
            b = old[comp] if not half else self.helm(old[comp], sp, comp)
            b = b + src
            if walls is not None and comp != 1:
                top, bot = (walls[0], walls[1]) if comp == 0 else (walls[2], walls[3])
                cw = 8.0 / 3.0 * n2 * ((sp - sm) if half else -sm)
                add = torch.zeros_like(b)
                add[:, 0, :] = cw * bot
                add[:, -1, :] = cw * top
                b = b + add
            if comp == 1:
                b = self.wallmask(b)
            new.append(self.helm_solve(b, sm, comp))
        return self.project(new)

    # markers -------------------------------------------------------------
    def _taps(self, X, comp):
        """Flat face indices and weights, [M, 64] (16 in 2D) each."""
        ext, idx, wt = (self.nx, self.ny, self.nz), [], []
        for a in range(3):
            if a == 2 and self.nz == 1:
                idx.append(torch.zeros((X.shape[0], 1), dtype=torch.int64, device=DEV))
                wt.append(torch.ones((X.shape[0], 1), dtype=torch.float64, device=DEV))
                continue
            t = X[:, a] * self.n - (0.0 if a == comp else 0.5)
            ft = torch.floor(t.detach())
            fr = (t - ft) * (math.pi / 2)
            S, C = torch.sin(fr), torch.cos(fr)
            wt.append(torch.stack([1 - S, 1 + C, 1 + S, 1 - C], 1) / 4)
            idx.append(torch.remainder(ft.to(torch.int64)[:, None] - 1 + torch.arange(4, device=DEV), ext[a]))
        i = idx[0][:, None, None, :] + self.nx * (idx[1][:, None, :, None] + self.ny * idx[2][:, :, None, None])
        w = wt[0][:, None, None, :] * wt[1][:, None, :, None] * wt[2][:, :, None, None]
        return i.reshape(X.shape[0], -1), w.reshape(X.shape[0], -1)

    def spread(self, X, F):
        sc = self.n ** (2 if self.nz == 1 else 3)
        out = []
        for comp in range(3):
            i, w = self._taps(X, comp)
            f = torch.zeros(self.nx * self.ny * self.nz, dtype=torch.float64, device=DEV)
            f = f.index_add(0, i.reshape(-1), (w * (sc * F[comp])[:, None]).reshape(-1))
            f = f.reshape(self.nz, self.ny, self.nx)
            out.append(self.wallmask(f) if comp == 1 else f)
        return out

    def interp(self, X, vel):
        out = []
        for comp in range(3):
            i, w = self._taps(X, comp)
            out.append((w * vel[comp].reshape(-1)[i]).sum(1))
        return torch.stack(out)

    def springs(self, X, lists, k, kb):
        rows, cols = lists

        def lap(Y):
            return torch.zeros_like(Y).index_add(0, rows, Y[cols] - Y[rows])
        Y = lap(X)
        G = k * Y
        if kb:
            G = G - kb * lap(Y)
        return G.T

    def ib_step(self, vel, X, lists, k, kb, dt):
        f = self.spread(X, self.springs(X, lists, k, kb))
        mid, _ = self.substep(vel, vel, f, False, None, None)
        Xh = X + dt / 2 * self.interp(X, mid).T
        U2 = self.interp(Xh, mid)
        f = self.spread(Xh, self.springs(Xh, lists, k, kb))
        new, _ = self.substep(vel, mid, f, True, None, None)
        return new, X + dt * U2.T


def _lists(nstart, nidx):
    rows = torch.from_numpy(np.repeat(np.arange(len(nstart) - 1), np.diff(nstart)).astype(np.int64)).to(DEV)
    return rows, torch.from_numpy(nidx.astype(np.int64)).to(DEV)


def exact(case, seed):
    kind = case["kind"]
    if _cells(case) > 300 ** 3:
        return None  # the spectral solves and the tap lists of 512^3 take too long
    E = _Exact(case)
    if kind in ("ib", "gradient"):
        Xn, nstart, nidx = _membrane(case, seed)
        X, lists = torch.from_numpy(Xn).to(DEV), _lists(nstart, nidx)
        vel, _ = E.project([E.full(a) for a in _flat(case, _random_velocity(case, seed))])
        if kind == "ib":
            with torch.no_grad():
                vel, X = E.ib_step(vel, X, lists, case["k"], case["kb"], case["dt"])
            return [E.flat(a) for a in vel] + [X]
        k = torch.tensor(case["k"], dtype=torch.float64, device=DEV, requires_grad=True)
        X0 = X.clone().requires_grad_(True)
        Y = X0
        for _ in range(case["steps"]):
            vel, Y = E.ib_step(vel, Y, lists, k, 0.0, case["dt"])
        uN = torch.stack([E.flat(a) for a in vel])
        membrane_like = (Y - Y.mean(0)) - (X - X.mean(0))
        ((membrane_like ** 2).sum() + 0.5 / float(_n(case)) ** 3 * (uN * uN).sum()).backward()
        return [uN.detach(), Y.detach(), k.grad, X0.grad]
    if kind == "ns":
        vel, g = E.project([E.full(a) for a in _flat(case, _random_velocity(case, seed))])
        f = [E.full(a) for a in _forces(case, seed)]
        walls = [a.reshape(E.nz, E.nx) for a in _walls(case, seed)] if E.ch else None
        old = vel
        for half in (False, True):
            vel, g = E.substep(old, vel, f, half, walls, g)
        return [E.flat(a, c) for c, a in enumerate(vel)]
    if kind == "project":
        vel, _ = E.project([E.full(a) for a in _flat(case, _provisional(case, seed))])
        return [E.flat(a, c) for c, a in enumerate(vel)]
    if kind == "helmholtz":
        _, b = _viscous_inputs(case, seed)
        return [E.flat(E.helm_solve(E.full(b), _scale(case), case["comp"]), case["comp"])]
    if kind == "transfers":
        X = torch.from_numpy(_membrane(case, seed)[0]).to(DEV)
        F = _marker_forces(case, X, seed)
        vel = [E.full(a) for a in _flat(case, _random_velocity(case, seed))]
        return [E.flat(a, c) for c, a in enumerate(E.spread(X, F))] + [E.interp(X, vel)]
    a = [E.full(t) for t in _operator_inputs(case, seed)]
    if case["op"] == "advection":
        return [E.flat(t, c) for c, t in enumerate(E.advection(*a))]
    if case["op"] == "laplacian":
        return [E.flat(E.lap(a[0]))]
    if case["op"] == "helmholtz":
        return [E.flat(E.helm(a[0], -0.1 / float(_n(case)) ** 2, 0))]
    if case["op"] == "divergence":
        return [E.flat(E.div(*a))]
    return [E.flat(t, c) for c, t in enumerate(E.grad(a[0]))]
