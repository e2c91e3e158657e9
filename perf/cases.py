"""What this framework's speed is measured on: whole calls through its public entry points.

Every case is a run that a user of the solver makes: an initial state handed over (or
built on the device), a number of time steps, and the state (or the gradients) back.
Sizes and states are those of the repository's own workloads (the N = 1000 Riemann
problem, the piecewise-constant segments, the uneven batch, the two-phase interface and
tanh profiles, the 65,536-cell adjoint), shortened to a few to a hundred steps so that
one pass is one call; `draw` spreads the same kinds over their whole range.

`exact` steps the same problem in plain torch, 64 bits throughout: the acoustic tensor
is differentiated by a complex step, gradients come from autograd.
"""
import ctypes
import math

import numpy as np
import torch

from hyperelasticsolver_gb300 import Barton2009, Batch, Hyperelasticity, HyperelasticityMPh, NumFluxes, Solver
from hyperelasticsolver_gb300 import _cases as C
from hyperelasticsolver_gb300 import _lib as L
from hyperelasticsolver_gb300 import _model as M

B0_SOFT = 2.1 * math.sqrt(0.1)  # phase 2 of the two-phase workload: a tenth of phase 1's shear modulus

# Floating-point operations per cell and step of the closed forms (multiply and add count
# one each): the counts of tests/test_flop_count.py for the Rusanov and HLL steps; LxF has
# 6 of HLL's 18 evaluations of the non-conservative matrix and no midpoint speeds; the
# adjoint's reverse step recomputes the forward one and costs about three times its flops.
FLOPS_1PH, FLOPS_HLL, FLOPS_LXF = 674, 15087, 5700


def listed():
    return [
        # The reference's own kind of run: a 1D Riemann problem of 1000 cells, FP64, to
        # and from host arrays. Latency and launches count here.
        dict(name="riemann_1000", kind="single", precision="fp64", flux="rusanov", bc="transmissive", data="riemann",
             n=1000, steps=100),
        # The smallest call: a caller with its own device memory advances its state a few
        # steps at a time in place of its own loop's body.
        dict(name="device_8192", kind="device", flux="rusanov", bc="frozen", n=8192, steps=4),
        # A resolved FP64 run, an odd number of cells, page-locked host arrays.
        dict(name="segments_1m", kind="single", precision="fp64", flux="rusanov", bc="frozen", data="segments",
             n=1000003, steps=10),
        # The mixed-precision production step.
        dict(name="segments_4m_mixed", kind="single", precision="mixed", flux="rusanov", bc="frozen",
             data="segments", n=1 << 22, steps=50),
        # Parameter studies: many problems of uneven size advanced together, both precisions.
        dict(name="batch_512_mixed", kind="batch", precision="mixed", flux="rusanov", problems=512, lo=256, hi=65536,
             steps=20),
        dict(name="batch_96", kind="batch", precision="fp64", flux="rusanov", problems=96, lo=256, hi=65536, steps=10),
        # main.jl as it stands: two phases, path-conservative HLL, a test-case Riemann problem.
        dict(name="two_riemann_1000", kind="two", precision="fp64", flux="hll", data="riemann", n=1000, steps=50),
        # main.jl's tanh profile (volume fractions vary in every cell), large and odd.
        dict(name="two_tanh_100k", kind="two", precision="fp64", flux="hll", data="tanh", n=100003, steps=4),
        # The smoothed-interface workload with the Lax-Friedrichs flux of main.jl:223.
        dict(name="two_interface_lxf", kind="two", precision="fp64", flux="lxf", data="interface", n=1 << 17, steps=4),
        # The same workload, HLL, in mixed precision.
        dict(name="two_interface_1m_mixed", kind="two", precision="mixed", flux="hll", data="interface", n=1 << 20,
             steps=10),
        # Gradient of a profile misfit with respect to the initial state and the moduli:
        # record, misfit, reverse pass.
        dict(name="adjoint_65536", kind="adjoint", n=65536, steps=50, ckpt=25),
        # The function-level API on arrays of faces.
        dict(name="faces_4096", kind="faces", n=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "device", "batch", "two", "two", "adjoint", "faces"])
    if kind == "single":
        precision = rng.choice(["fp64", "fp64", "mixed"])
        n = _log_int(rng, 300, 1000000 if precision == "fp64" else 4000000)
        steps = max(1, min(100, _log_int(rng, 4, 40), (10000000 if precision == "fp64" else 200000000) // n))
        return dict(kind=kind, precision=precision, flux=rng.choice(["rusanov", "rusanov", "lxf"]),
                    bc=rng.choice(["frozen", "transmissive"]), data=rng.choice(["riemann", "segments"]), n=n,
                    steps=steps)
    if kind == "device":
        return dict(kind=kind, flux=rng.choice(["rusanov", "lxf"]), bc=rng.choice(["frozen", "transmissive"]),
                    n=_log_int(rng, 200, 65536), steps=rng.randint(1, 8))
    if kind == "batch":
        return dict(kind=kind, precision=rng.choice(["fp64", "mixed"]), flux=rng.choice(["rusanov", "rusanov", "lxf"]),
                    problems=_log_int(rng, 8, 96), lo=256, hi=rng.choice([4096, 65536]), steps=rng.randint(4, 10))
    if kind == "two":
        precision = rng.choice(["fp64", "fp64", "mixed"])
        n = _log_int(rng, 300, 100000 if precision == "fp64" else 1000000)
        steps = max(1, min(_log_int(rng, 2, 40), (400000 if precision == "fp64" else 10000000) // n))
        return dict(kind=kind, precision=precision, flux=rng.choice(["hll", "hll", "lxf"]),
                    data=rng.choice(["riemann", "tanh", "interface"]), n=n, steps=steps)
    if kind == "adjoint":
        n = _log_int(rng, 500, 65000)
        return dict(kind=kind, n=n, steps=rng.randint(10, 50), ckpt=rng.randint(5, 50))
    return dict(kind=kind, n=_log_int(rng, 1, 4096))


def work(case):
    """Each step reads and writes the whole state once (the global maximum wave speed
    stands between two steps); transfers to and from the host are the state once each way."""
    k, steps = case["kind"], case.get("steps", 1)
    if k == "faces":
        return {"bytes": (5 * 30 + 1) * 8 * case["n"], "flops": FLOPS_LXF * case["n"]}
    if k == "batch":
        n, row, f = int(_batch_sizes(case).sum()), 14 * 8, FLOPS_1PH
    elif k == "two":
        n, row, f = case["n"], 30 * 8, FLOPS_LXF if case["flux"] == "lxf" else FLOPS_HLL
    else:
        n, row, f = case["n"], 14 * 8, FLOPS_1PH
    if k == "adjoint":  # forward, recompute, and the reverse steps
        return {"bytes": 3 * 2 * row * n * steps, "flops": 5 * f * n * steps}
    return {"bytes": 2 * row * n * steps, "flops": f * n * steps}


# ---- inputs -----------------------------------------------------------------


def _batch_sizes(case):
    return C.batch_sizes(case["problems"], case["lo"], case["hi"], seed=C.SEGMENT_SEED)


def _eos2():
    return Barton2009(), Barton2009(_b0=B0_SOFT)


def _riemann_prims(eos, seed):
    """The config-1 Riemann states with a jitter from the seed (one problem of C.batch_prims)."""
    l, r = C.batch_prims(eos, 1, seed=seed)
    return l[0], r[0]


def _single_prims(case, seed):
    """Primitive states (k, 14) and, per cell, which of them it carries."""
    eos, n = Barton2009(), case["n"]
    if case.get("data", "segments") == "riemann":
        return np.stack(_riemann_prims(eos, seed)), (np.arange(n) >= n / 2).astype(np.int64)
    return C.segment_states(eos, seed=seed), (np.arange(n, dtype=np.int64) * 64) // n


def _two_prims(case, seed):
    """Left and right primitive 30-vectors of a two-phase case."""
    rng = np.random.default_rng(seed)
    if case["data"] == "interface":  # both phases in the single-phase Riemann states
        l, r = _riemann_prims(Barton2009(), seed)
        return np.concatenate([[1.0], l, [1.0], l]), np.concatenate([[1.0], r, [1.0], r])
    l, r = C.mph_case(6)  # main.jl's Riemann test cases: volume fractions 0.1 | 0.9
    s = rng.uniform(0.8, 1.2)
    for p in (l, r):
        p[2:5] *= s
        p[17:20] *= s
    return l, r


def _alpha1(case, eps):
    """Volume fraction of phase 1 per cell."""
    n = case["n"]
    x = (np.arange(n) + 0.5) / n
    if case["data"] == "tanh":
        return 0.1 * (np.tanh(4.0 * (x - 0.5) / eps) + 1.0) + 0.4
    return 1e-6 + (1.0 - 2e-6) * 0.5 * (1.0 - np.tanh(4.0 * (x - 0.5) * n / 8.0))


class State:
    pass


TANH_EPS = 0.2


def _pinned(shape):
    """Page-locked host memory as a numpy array."""
    return torch.empty(tuple(shape), dtype=torch.float64, pin_memory=True).numpy()


def _pin(a):
    p = _pinned(a.shape)
    p[...] = a
    return p


def prepare(case, seed):
    s = State()
    s.case, kind = dict(case), case["kind"]
    if kind == "single":
        eos = Barton2009()
        prims, which = _single_prims(case, seed)
        s.Q = _pin(Hyperelasticity.prim2cons(eos, prims).T[:, which])
        s.out = _pinned(s.Q.shape)
        s.solver = Solver(eos, case["n"], flux=case["flux"], bc=case["bc"], precision=case["precision"])
    elif kind == "device":
        eos = Barton2009()
        prims, which = _single_prims(case, seed)
        s.Q = torch.from_numpy(np.ascontiguousarray(Hyperelasticity.prim2cons(eos, prims).T[:, which])).cuda()
        s.out = torch.empty_like(s.Q)
        flux = {"rusanov": L.HYP_FLUX_RUSANOV, "lxf": L.HYP_FLUX_LXF}[case["flux"]]
        bc = {"frozen": L.HYP_BC_FROZEN, "transmissive": L.HYP_BC_TRANSMISSIVE}[case["bc"]]
        s.cfg = M.config(eos, L.HYP_MODEL_SINGLE, case["n"], flux, bc)
        s.step = L.load().hyp_step_noalloc_f64
    elif kind == "batch":
        eos, sizes = Barton2009(), _batch_sizes(case)
        l, r = C.batch_prims(eos, len(sizes), seed=seed)
        s.Q = _pin(C.batch_fill(Hyperelasticity.prim2cons(eos, l), Hyperelasticity.prim2cons(eos, r), sizes))
        s.out = _pinned(s.Q.shape)
        s.batch = Batch(eos, sizes, flux=case["flux"], precision=case["precision"])
    elif kind == "two":
        eos, n = _eos2(), case["n"]
        Pl, Pr = _two_prims(case, seed)
        s.Ql, s.Qr = HyperelasticityMPh.prim2cons_mph(eos, np.stack([Pl, Pr]))
        if case["data"] == "interface":
            a1 = _alpha1(case, TANH_EPS)
            alpha = np.concatenate([np.tile(a1, (15, 1)), np.tile(1.0 - a1, (15, 1))])
            s.Q = _pin(C.initial_condition(s.Ql, s.Qr, n) * alpha)
        s.out = _pinned((30, n))
        s.solver = Solver(eos, n, model="multi", flux=case["flux"], precision=case["precision"])
    elif kind == "adjoint":
        eos, n = Barton2009(), case["n"]
        prims, which, s.target = _adjoint_inputs(case, seed)
        s.Q = Hyperelasticity.prim2cons(eos, prims).T[:, which].copy()
        s.solver = Solver(eos, n)
    else:
        l, r = _face_prims(case, seed)
        s.eos = _eos2()
        s.Ql = HyperelasticityMPh.prim2cons_mph(s.eos, l)
        s.Qr = HyperelasticityMPh.prim2cons_mph(s.eos, r)
        s.lam = _face_speeds(case, seed)
    return s


def _adjoint_inputs(case, seed):
    """The adjoint workload's Riemann states with a jitter, and a measured density profile
    to fit: the initial one smeared over the domain's middle, with 1 % noise."""
    rng = np.random.default_rng(seed)
    eos, n = Barton2009(), case["n"]
    l, r = C.adjoint_states(eos)
    for p in (l, r):
        p[1:4] *= rng.uniform(0.9, 1.1)
    x = (np.arange(n) + 0.5) / n
    w = 0.5 * (1.0 + np.tanh((x - 0.5) / 0.05))
    target = (l[0] * (1.0 - w) + r[0] * w) * (1.0 + 0.01 * rng.standard_normal(n))
    return np.stack([l, r]), (np.arange(n) >= n / 2).astype(np.int64), target


def _face_prims(case, seed):
    """Left and right primitive states of independent faces (n, 30): alpha1 in
    (0.05, 0.95), a strain and a velocity per phase; the right state near the left."""
    rng, n = np.random.default_rng(seed), case["n"]
    out = []
    F0 = np.eye(3) + 0.02 * rng.standard_normal((n, 2, 3, 3))
    u0 = rng.uniform(-0.4, 0.4, (n, 2, 3))
    a0 = rng.uniform(0.1, 0.9, n)
    for _ in range(2):
        F = F0 + 0.02 * rng.standard_normal((n, 2, 3, 3))
        u = u0 + rng.uniform(-0.2, 0.2, (n, 2, 3))
        a = a0 + rng.uniform(-0.05, 0.05, n)
        P = np.empty((n, 30))
        for p in range(2):
            P[:, 15 * p] = a if p == 0 else 1.0 - a
            P[:, 15 * p + 1] = 8.93 / np.linalg.det(F[:, p])
            P[:, 15 * p + 2:15 * p + 5] = u[:, p]
            P[:, 15 * p + 5] = rng.uniform(0.0, 5e-4, n)
            P[:, 15 * p + 6:15 * p + 15] = F[:, p].transpose(0, 2, 1).reshape(n, 9)
        out.append(P)
    return out


def _face_speeds(case, seed):
    return np.random.default_rng(seed + 1).uniform(5.0, 8.0, case["n"])


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "single":
        s.solver.upload(s.Q)
        steps, t = s.solver.step(case["steps"])
        return {"Q": s.solver.download(s.out), "t": t, "steps": steps}
    if kind == "device":
        t, bad = ctypes.c_double(0.0), ctypes.c_int64(-1)
        L.check(s.step(s.cfg, s.Q.data_ptr(), s.out.data_ptr(), case["n"], case["steps"], 0.0,
                       torch.cuda.current_stream().cuda_stream, ctypes.byref(t), ctypes.byref(bad)),
                what="hyp_step_noalloc_f64")
        return {"Q": s.out, "t": t.value}
    if kind == "batch":
        s.batch.upload(s.Q)
        s.batch.step(case["steps"])
        t, steps = s.batch.status()
        return {"Q": s.batch.download(s.out), "t": t, "steps": steps}
    if kind == "two":
        if case["data"] == "riemann":
            s.solver.init_riemann(s.Ql, s.Qr)
        elif case["data"] == "tanh":
            s.solver.init_tanh(s.Ql, s.Qr, TANH_EPS)
        else:
            s.solver.upload(s.Q)
        steps, t = s.solver.step(case["steps"])
        return {"Q": s.solver.download(s.out), "t": t, "steps": steps}
    if kind == "adjoint":
        s.solver.upload(s.Q)
        t = s.solver.record(case["steps"], case["ckpt"])
        loss, dQ = s.solver.density_misfit(s.target)
        dQ0, deos = s.solver.adjoint(dQ)
        return {"loss": loss, "dQ": dQ, "dQ0": dQ0, "deos": deos, "t": t}
    cons, dm, dp = NumFluxes.lxf(s.eos, s.Ql, s.Qr, s.lam)
    return {"cons": cons, "dm": dm, "dp": dp}


# ---- the same in plain torch, 64 bits ---------------------------------------


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Eos:
    def __init__(self, e, b0sq=None, k0=None):
        self.rho0, self.cv, self.t0, self.al, self.be, self.ga = e.rho0, e.cv, e.t0, e.alpha, e.beta, e.gamma
        self.b0sq = e.b0sq if b0sq is None else b0sq
        self.k0 = e.k0 if k0 is None else k0


def _det(A):
    return (A[..., 0] * torch.linalg.cross(A[..., 1], A[..., 2], dim=-1)).sum(-1)


def _strain(A):
    """G = (A A^T)^-1, its first two invariants and det G."""
    m = A @ A.transpose(-1, -2)
    p = 1.0 / _det(A) ** 2
    G = torch.stack([torch.linalg.cross(m[..., 1], m[..., 2], dim=-1), torch.linalg.cross(m[..., 2], m[..., 0], dim=-1),
                     torch.linalg.cross(m[..., 0], m[..., 1], dim=-1)], -1) * p[..., None, None]
    i1 = G.diagonal(dim1=-2, dim2=-1).sum(-1)
    i2 = 0.5 * (i1 * i1 - (G @ G).diagonal(dim1=-2, dim2=-1).sum(-1))
    return G, i1, i2, p


def _x(e, eint, A):
    """The argument of the entropy's logarithm: exp(S / cv)."""
    _, i1, i2, p = _strain(A)
    cold = 0.5 * e.k0 / e.al ** 2 * (p ** (0.5 * e.al) - 1.0) ** 2
    shear = 0.5 * e.b0sq * p ** (0.5 * e.be) * (i1 * i1 / 3.0 - i2)
    return ((eint - shear - cold) / (e.cv * e.t0 * p ** (0.5 * e.ga)) + 1.0).clamp(min=1e-6)


def _energy(e, x, A):
    _, i1, i2, p = _strain(A)
    return (0.5 * e.k0 / e.al ** 2 * (p ** (0.5 * e.al) - 1.0) ** 2 + e.cv * e.t0 * p ** (0.5 * e.ga) * (x - 1.0)
            + 0.5 * e.b0sq * p ** (0.5 * e.be) * (i1 * i1 / 3.0 - i2))


def _sigma0(e, x, A):
    """First row of the stress over the density: -2 G dE/dG at fixed entropy."""
    G, i1, i2, p = _strain(A)
    pb = p ** (0.5 * e.be)
    e1, e2 = e.b0sq / 3.0 * pb * i1, -0.5 * e.b0sq * pb
    pa = p ** (0.5 * e.al)
    e3p = (0.5 * e.k0 / e.al * (pa - 1.0) * pa + 0.5 * e.cv * e.t0 * e.ga * p ** (0.5 * e.ga) * (x - 1.0)
           + 0.25 * e.b0sq * e.be * pb * (i1 * i1 / 3.0 - i2))
    g0 = G[..., 0, :]
    h0 = (g0[..., None, :] @ G)[..., 0, :]
    one = torch.zeros(3, dtype=A.dtype, device=A.device)
    one[0] = 1.0
    return -2.0 * ((e1 + e2 * i1)[..., None] * g0 - e2[..., None] * h0 + e3p[..., None] * one)


def _top_eigenvalue(a):
    """Largest eigenvalue of symmetric 3x3 matrices: the trigonometric root of the
    characteristic polynomial, then Newton steps; the last one carries the derivative."""
    c2 = a.diagonal(dim1=-2, dim2=-1).sum(-1)
    c1 = 0.5 * (c2 * c2 - (a * a).sum((-2, -1)))
    c0 = _det(a)
    with torch.no_grad():
        q = c2 / 3.0
        b = a - q[..., None, None] * torch.eye(3, dtype=a.dtype, device=a.device)
        p = torch.sqrt((b * b).sum((-2, -1)) / 6.0).clamp(min=1e-300)
        r = q + 2.0 * p * torch.cos(torch.acos((0.5 * _det(b) / p ** 3).clamp(-1.0, 1.0)) / 3.0)
    for k in range(3):
        r = r.detach()
        r = r - (((r - c2) * r + c1) * r - c0) / ((3.0 * r - 2.0 * c2) * r + c1).detach()
    return r


def _phase(e, q):
    """One phase's primitives, first stress row, largest acoustic speed and temperature.
    q: the 15 values (alpha, alpha rho, alpha rho u, alpha rho E, alpha rho A), last axis."""
    a, m, rE = q[..., 0], q[..., 2:5], q[..., 5]
    rA = q[..., 6:15].reshape(q.shape[:-1] + (3, 3)).transpose(-1, -2)
    rho = torch.sqrt(_det(rA / a[..., None, None]) / e.rho0)
    den = a * rho
    u, E, A = m / den[..., None], rE / den, rA / den[..., None, None]
    eint = E - 0.5 * (u * u).sum(-1)
    x = _x(e, eint, A)
    dens = e.rho0 / _det(A)
    s0 = _sigma0(e, x, A)
    h = 1e-20
    cols = []
    for j in range(3):  # d sigma_0i / dA along e_j A[0, :], the entropy held
        d = torch.zeros_like(A)
        d[..., j, :] = A[..., 0, :]
        Z = torch.complex(A, h * d)
        cols.append((_sigma0(e, x, Z) / _det(Z)[..., None]).imag / h * _det(A)[..., None])
    om = torch.stack(cols, -1)
    c = torch.sqrt(_top_eigenvalue(0.5 * (om + om.transpose(-1, -2))))
    T = _strain(A)[3] ** (0.5 * e.ga) * e.t0 * x
    return dict(a=a, den=den, rho=rho, u=u, E=E, S=e.cv * torch.log(x), A=A, s0=dens[..., None] * s0, c=c, T=T)


def _flux(f):
    s = f["s0"] * f["a"][..., None]
    du = f["den"] * f["u"][..., 0]
    mom = du[..., None] * f["u"] - s
    en = du * f["E"] - (f["u"] * s).sum(-1)
    A, u = f["A"], f["u"]
    rA = f["den"][..., None, None] * (u[..., 0, None, None] * A - u[..., :, None] * A[..., None, 0, :])
    rA = rA.transpose(-1, -2).reshape(rA.shape[:-2] + (9,))
    return torch.cat([torch.zeros_like(du)[..., None], du[..., None], mom, en[..., None], rA], -1)


def _noncons(f):
    """Column of the non-conservative matrix for each phase (alpha's own column)."""
    b1, b2 = f
    uI = 0.5 * (b1["u"] + b2["u"])
    sI = (b2["T"][..., None] * b1["s0"] + b1["T"][..., None] * b2["s0"]) / (b1["T"] + b2["T"])[..., None]
    out = []
    for b in f:
        rA = b["rho"][..., None, None] * b["u"][..., :, None] * b["A"][..., None, 0, :]
        row0 = b["rho"][..., None] * (b["A"] * (uI - b["u"])[..., :, None]).sum(-2)
        rA = torch.cat([rA[..., :1, :] + row0[..., None, :], rA[..., 1:, :]], -2)
        out.append(torch.cat([uI[..., :1], torch.zeros_like(uI[..., :1]), sI, (sI * uI).sum(-1, keepdim=True),
                              rA.transpose(-1, -2).reshape(uI.shape[:-1] + (9,))], -1))
    return torch.cat(out, -1)


def _both(eos, Q):
    return [_phase(eos[0], Q[..., :15]), _phase(eos[1], Q[..., 15:])]


def _speeds(f):
    lo = torch.minimum(f[0]["u"][..., 0] - f[0]["c"], f[1]["u"][..., 0] - f[1]["c"])
    hi = torch.maximum(f[0]["u"][..., 0] + f[0]["c"], f[1]["u"][..., 0] + f[1]["c"])
    return lo, hi


def _nodes(flux):
    if flux == "hll":
        x, w = np.polynomial.legendre.leggauss(6)
    else:
        p5 = np.polynomial.legendre.Legendre.basis(5)
        x = np.concatenate([[-1.0], np.sort(p5.deriv().roots().real), [1.0]])
        w = 2.0 / (30.0 * p5(x) ** 2)
    return 0.5 * (x + 1.0), 0.5 * w


def _path(eos, flux, Qa, Qb):
    d = Qb - Qa
    da = torch.cat([d[..., :1].expand(d.shape[:-1] + (15,)), d[..., 15:16].expand(d.shape[:-1] + (15,))], -1)
    acc = torch.zeros_like(Qa)
    for x, w in zip(*_nodes(flux)):
        acc = acc + float(w) * _noncons(_both(eos, Qa * (1.0 - float(x)) + Qb * float(x))) * da
    return acc


def _hll(eos, QL, QR, fL, fR, lo, hi):
    ml, mh = _speeds(_both(eos, 0.5 * (QL + QR)))
    sl = torch.minimum(ml, lo).clamp(max=0.0)[..., None]
    sr = torch.maximum(mh, hi).clamp(min=0.0)[..., None]
    Qh = ((QR * sr - QL * sl) - (_path(eos, "hll", QL, QR) + fR - fL)) / (sr - sl)
    inner = fR - fL + _path(eos, "hll", QL, Qh) + _path(eos, "hll", Qh, QR)
    cq = sl * sr / (sr - sl) * (QR - QL)
    return -sl / (sr - sl) * inner + cq, sr / (sr - sl) * inner - cq


def _in_parts(f, Q, most=1 << 17):
    """f over the rows of Q in parts, to bound the working set."""
    return torch.cat([f(Q[i:i + most]) for i in range(0, Q.shape[0], most)])


def _step_single(e, Q, dx, flux, bc, prob=None, first=None, last=None):
    """One step of 14-value cells Q (n, 14); with `prob` (problem of each cell) a batch.
    Returns the new cells and each problem's dt."""
    def cell(q):
        f = _phase(e, torch.cat([torch.ones_like(q[:, :1]), q], -1))
        return torch.cat([_flux(f)[:, 1:], (f["u"][:, 0].abs() + f["c"])[:, None]], -1)

    fl = _in_parts(cell, Q) if not Q.requires_grad else cell(Q)
    F, lam = fl[:, :14], fl[:, 14]
    n = Q.shape[0]
    if prob is None:
        dt = 0.5 * dx / lam[(lam == lam.max()).nonzero()[0, 0]]
        r = dt / dx
        ends = torch.zeros(n, dtype=torch.bool, device=Q.device)
        ends[0] = ends[-1] = True
        left = torch.cat([torch.zeros(1, dtype=torch.long, device=Q.device), torch.arange(n - 1, device=Q.device)])
        right = torch.cat([torch.arange(1, n, device=Q.device), torch.tensor([n - 1], device=Q.device)])
        lf = dx / dt
    else:
        top = torch.zeros(len(dx), dtype=Q.dtype, device=Q.device).scatter_reduce(0, prob, lam, "amax")
        dt = 0.5 * dx / top
        r = (dt / dx)[prob][:, None]
        lf = (dx / dt)[prob]
        i = torch.arange(n, device=Q.device)
        ends = first | last
        left, right = torch.where(first, i, i - 1), torch.where(last, i, i + 1)

    def face(a, b):
        s = torch.maximum(lam[a], lam[b]) if flux == "rusanov" else lf
        s = s[:, None] if torch.is_tensor(s) and s.dim() else s
        return 0.5 * (F[a] + F[b]) - 0.5 * s * (Q[b] - Q[a])

    i = torch.arange(n, device=Q.device)
    new = Q - r * (face(i, right) - face(left, i))
    return (torch.where(ends[:, None], Q, new) if bc == "frozen" else new), dt


def _step_two(eos, Q, dx, flux):
    def cell(q):
        f = _both(eos, q)
        return torch.cat([_flux(f[0]), _flux(f[1]), torch.stack(_speeds(f), -1)], -1)

    out = _in_parts(cell, Q)
    F, lo, hi = out[:, :30], out[:, 30], out[:, 31]
    dt = 0.5 * dx / torch.maximum(lo.abs(), hi.abs()).max()
    lf = dx / dt

    def face(x):
        QL, QR, fL, fR, a, b = x[:, :30], x[:, 30:60], x[:, 60:90], x[:, 90:120], x[:, 120], x[:, 121]
        if flux == "hll":
            return torch.cat(_hll(eos, QL, QR, fL, fR, a, b), -1)
        cons, half = 0.5 * (fL + fR) - 0.5 * lf * (QR - QL), 0.5 * _path(eos, "lxf", QL, QR)
        return torch.cat([cons + half, half - cons], -1)

    d = _in_parts(face, torch.cat([Q[:-1], Q[1:], F[:-1], F[1:], lo[:-1, None], hi[1:, None]], -1), 1 << 15)
    new = Q.clone()
    new[1:-1] = Q[1:-1] - dt / dx * (d[1:, :30] + d[:-1, 30:])
    return new, dt


def _cons(e, prims):
    """Single-phase conservative states (k, 14) of primitive ones (rho, u, S, A)."""
    P = torch.as_tensor(np.asarray(prims), dtype=torch.float64, device=_dev())
    A = P[:, 5:14].reshape(-1, 3, 3).transpose(-1, -2)
    E = _energy(e, torch.exp(P[:, 4] / e.cv), A) + 0.5 * (P[:, 1:4] ** 2).sum(-1)
    return torch.cat([P[:, :1], P[:, :1] * P[:, 1:4], (P[:, 0] * E)[:, None], P[:, :1] * P[:, 5:14]], -1)


def _prims2(eos, Q):
    """Primitive 30-vectors of conservative ones: the density is the one that det(rho A) gives."""
    out = []
    for f in _both(eos, Q):
        A = f["A"].transpose(-1, -2).reshape(f["A"].shape[:-2] + (9,))
        out.append(torch.cat([f["a"][..., None], f["rho"][..., None], f["u"], f["S"][..., None], A], -1))
    return torch.cat(out, -1)


def _cons2(eos, prims):
    P = np.asarray(prims)
    out = []
    for p, e in enumerate(eos):
        q = _cons(e, P[:, 15 * p + 1:15 * p + 15])
        a = torch.as_tensor(P[:, 15 * p:15 * p + 1], dtype=torch.float64, device=_dev())
        out.append(torch.cat([a, a * q], -1))
    return torch.cat(out, -1)


def exact(case, seed):
    kind, dev = case["kind"], _dev()
    if kind in ("single", "device"):
        e = _Eos(Barton2009())
        prims, which = _single_prims(case, seed)
        Q = _cons(e, prims)[torch.from_numpy(which).to(dev)]
        dx, t = 1.0 / case["n"], 0.0
        for _ in range(case["steps"] if case["n"] * case["steps"] <= 20000000 else 0):
            Q, dt = _step_single(e, Q, dx, case["flux"], case["bc"])
            t += float(dt)
        if t == 0.0:
            return None
        out = {"Q": Q.T.contiguous(), "t": t}
        return out if kind == "device" else dict(out, steps=None)
    if kind == "batch":
        e, sizes = _Eos(Barton2009()), _batch_sizes(case)
        if sizes.sum() * case["steps"] > 20000000:
            return None
        l, r = C.batch_prims(Barton2009(), len(sizes), seed=seed)
        both = torch.stack([_cons(e, l), _cons(e, r)])
        p = np.repeat(np.arange(len(sizes)), sizes)
        k = np.arange(len(p)) - np.repeat(np.cumsum(sizes) - sizes, sizes)
        prob = torch.from_numpy(p).to(dev)
        first, last = (torch.from_numpy(m).to(dev) for m in (k == 0, k == sizes[p] - 1))
        Q = both[torch.from_numpy((k >= sizes[p] / 2).astype(np.int64)).to(dev), prob]
        dx = 1.0 / torch.from_numpy(sizes.astype(np.float64)).to(dev)
        t = torch.zeros_like(dx)
        for _ in range(case["steps"]):
            Q, dt = _step_single(e, Q, dx, case["flux"], "frozen", prob, first, last)
            t = t + dt
        return {"Q": Q.T.contiguous(), "t": t, "steps": None}
    if kind == "two":
        if case["n"] * case["steps"] > 600000:
            return None
        eos, n = tuple(_Eos(e) for e in _eos2()), case["n"]
        Pl, Pr = _two_prims(case, seed)
        if case["data"] == "tanh":
            Pl, Pr = _prims2(eos, _cons2(eos, np.stack([Pl, Pr]))).cpu().numpy()
        # the two-state fill is by cell number, the tanh profile's by position: they differ in the middle cell of an odd n
        left = (np.arange(n) + 0.5) / n < 0.5 if case["data"] == "tanh" else np.arange(n) < n / 2
        P = np.where(left[:, None], Pl[None], Pr[None])
        if case["data"] != "riemann":
            a1 = _alpha1(case, TANH_EPS)
            P[:, 0], P[:, 15] = a1, 1.0 - a1
        Q, t = _cons2(eos, P), 0.0
        for _ in range(case["steps"]):
            Q, dt = _step_two(eos, Q, 1.0 / n, case["flux"])
            t += float(dt)
        return {"Q": Q.T.contiguous(), "t": t, "steps": None}
    if kind == "faces":
        eos = tuple(_Eos(e) for e in _eos2())
        QL, QR = (_cons2(eos, P) for P in _face_prims(case, seed))
        fL, fR = (torch.cat([_flux(p) for p in _both(eos, q)], -1) for q in (QL, QR))
        lam = torch.from_numpy(_face_speeds(case, seed)).to(dev)[:, None]
        half = 0.5 * _path(eos, "lxf", QL, QR)
        return {"cons": 0.5 * (fL + fR) - 0.5 * lam * (QR - QL), "dm": half, "dp": half}
    # adjoint: the steps forward, then autograd step by step backwards
    b = Barton2009()
    prims, which, target = _adjoint_inputs(case, seed)
    dx, t = 1.0 / case["n"], 0.0
    mod = [torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True) for v in (b.b0sq, b.k0)]
    e = _Eos(b, *mod)
    states = [_cons(_Eos(b), prims)[torch.from_numpy(which).to(dev)]]
    with torch.no_grad():
        for _ in range(case["steps"]):
            Q, dt = _step_single(e, states[-1], dx, "rusanov", "frozen")
            t += float(dt)
            states.append(Q)
    Q = states.pop().requires_grad_()
    rho = torch.sqrt(_det(Q[:, 5:14].reshape(-1, 3, 3)) / e.rho0)
    loss = 0.5 * ((rho - torch.from_numpy(target).to(dev)) ** 2).sum()
    g, = torch.autograd.grad(loss, Q)
    dQ, deos = g, torch.zeros(2, dtype=torch.float64, device=dev)
    while states:
        Q = states.pop().requires_grad_()
        new, _ = _step_single(e, Q, dx, "rusanov", "frozen")
        g, g0, g1 = torch.autograd.grad(new, [Q] + mod, g)
        deos = deos + torch.stack([g0, g1])
    return {"loss": float(loss.detach()), "dQ": dQ.T.contiguous(), "dQ0": g.T.contiguous(), "deos": deos, "t": t}
