"""The FP64 step's compact cell forms (hyp_cell64.cuh, host build) against the general
closed forms and the oracle: flux, wave speed and status. CPU only."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

from helpers import RTOL_FP64

HERE = os.path.dirname(os.path.abspath(__file__))
EOS = [(8.93, 4.6, 3.9e-4, 300, 2.1, 1, 3, 2), (8.93, 4.6, 3.9e-4, 300, 2.1 * 0.1 ** 0.5, 1, 3, 2),
       (8.93, 6.22, 9.0e-4, 300, 3.16, 1, 3.577, 2.088)]


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(tempfile.mkdtemp(prefix="hyp_c64_"), "c64.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                        os.path.join(HERE, "cell64_shim.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = ctypes.CDLL(so)
    L.c64_to_f32.restype, L.c64_to_f32.argtypes = ctypes.c_float, [ctypes.c_double]
    L.c64_to_f64.restype, L.c64_to_f64.argtypes = ctypes.c_double, [ctypes.c_float]
    return L


def ev(lib, name, ep, q):
    dp = ctypes.POINTER(ctypes.c_double)
    e, q, out = np.array(ep, dtype=np.float64), np.ascontiguousarray(q), np.zeros(16)
    return getattr(lib, name)(e.ctypes.data_as(dp), q.ctypes.data_as(dp), out.ctypes.data_as(dp)), out


def phase_states(orc, ep, rng, n, alphas, strain):
    pb = orc.problem(eos=(orc.barton2009(*ep),) * 2)
    out = []
    while len(out) < n:
        F = np.eye(3) + strain * rng.standard_normal((3, 3))
        if np.linalg.det(F) < 0.3:
            continue
        P = np.array([8.93 / np.linalg.det(F), *rng.uniform(-0.6, 0.6, 3), rng.uniform(0, 1e-3), *F.reshape(-1, order="F")])
        a = rng.choice(alphas)
        out.append(np.concatenate([[a], a * np.asarray(orc.prim2cons(pb, P)).reshape(-1)]))
    return out


@pytest.mark.parametrize("ep", EOS)
@pytest.mark.parametrize("strain", [0.0, 1e-6, 0.02, 0.1, 0.25])
def test_compact_matches_general_and_oracle(lib, orc, ep, strain):
    """Both evaluate the same expression in another order; each component is held to the
    FP64 parity tolerance of the largest component of its kind (flux parts scale with
    alpha; a phase at alpha = 1e-6 is included)."""
    rng = np.random.default_rng(3)
    pb = orc.problem(eos=(orc.barton2009(*ep),) * 2)
    for q in phase_states(orc, ep, rng, 60, (1.0, 0.5, 0.03, 1e-6), strain):
        s0, g = ev(lib, "c64_general", ep, q)
        s1, c = ev(lib, "c64_compact", ep, q)
        assert s0 == s1 == 0
        f = np.asarray(orc.flux(pb, q[1:] / q[0])).reshape(-1) * q[0]
        lam = np.max(np.abs(orc.speeds(pb, q[1:] / q[0])))
        for ref in (g, np.concatenate([f, [g[14]], [lam - abs(g[14])]])):
            assert np.max(np.abs(c[:14] - ref[:14])) <= RTOL_FP64 * np.max(np.abs(ref[:14]))
            assert abs(c[14] - ref[14]) <= RTOL_FP64 * max(abs(ref[14]), 1e-300)
            assert abs(c[15] - ref[15]) <= RTOL_FP64 * (abs(ref[15]) + abs(ref[14]))


@pytest.mark.parametrize("ep", EOS)
def test_far_states_and_status(lib, orc, ep):
    """States off the ordinary path: close wave speeds (sheared or strongly stretched), the
    clamped entropy argument, det <= 0, NaN and infinities: same status, same values."""
    rng = np.random.default_rng(4)
    base = phase_states(orc, ep, rng, 1, (0.4,), 0.05)[0]
    cases = []
    for k in range(300):  # strong stretches along each axis: the spectrum's top root crosses others
        F = np.diag(np.exp(rng.uniform(-1.0, 1.0, 3))) + 0.2 * rng.standard_normal((3, 3))
        if np.linalg.det(F) < 0.05:
            continue
        a, rho = 0.4, 8.93 / np.linalg.det(F)
        cases.append(np.concatenate([[a, a * rho], a * rho * rng.uniform(-1, 1, 3), [a * rho * rng.uniform(-2, 60)],
                                     a * rho * F.reshape(-1, order="F")]))
    for j, v in ((5, -1e3), (5, np.nan), (6, -10.0), (6, np.inf), (10, 0.0), (3, np.nan), (5, np.inf), (8, np.nan)):
        q = base.copy()
        q[j] = v
        cases.append(q)
    cases.append(np.concatenate([base[:6], np.zeros(9)]))
    for q in cases:
        s0, g = ev(lib, "c64_general", ep, q)
        s1, c = ev(lib, "c64_compact", ep, q)
        assert s0 == s1, (q, s0, s1)
        if s0 == 0:
            assert np.all(np.isfinite(g) == np.isfinite(c))
            if np.all(np.isfinite(g)):
                # the energy-like terms cancel at these strains: compare on their scale
                scale = np.max(np.abs(g)) * max(1.0, np.linalg.cond(q[6:].reshape(3, 3)) ** 2)
                assert np.max(np.abs(g - c)) <= RTOL_FP64 * scale


@pytest.mark.parametrize("ep", EOS)
@pytest.mark.parametrize("strain", [0.0, 0.02, 0.1, 0.4])
@pytest.mark.parametrize("seeds", ["flux", "speed", "both"])
def test_vjp_matches_general(lib, orc, ep, strain, seeds):
    """The compact cell VJP against the general one, over seeds of the flux, the wave speed
    and both; strain 0.4 includes cells whose wave speeds are close (the general route)
    and states at the entropy clamp. Each is a sum of products whose factors reach
    |dF/dq| max|F-bar|: held to the parity tolerance of the largest entry."""
    rng = np.random.default_rng(9)
    dp = ctypes.POINTER(ctypes.c_double)
    e = np.array(ep, dtype=np.float64)
    for i, s in enumerate(phase_states(orc, ep, rng, 60, (1.0,), strain)):
        q = np.ascontiguousarray(s[1:])
        if i % 7 == 3:
            q[4] -= 3.0 * q[0]  # below the clamp
        fb = rng.standard_normal(14) if seeds != "speed" else np.zeros(14)
        lb = ctypes.c_double(rng.standard_normal() if seeds != "flux" else 0.0)
        out = [np.zeros(16), np.zeros(16)]
        st = [getattr(lib, n)(e.ctypes.data_as(dp), q.ctypes.data_as(dp), fb.ctypes.data_as(dp), lb, o.ctypes.data_as(dp))
              for n, o in zip(("c64_vjp_general", "c64_vjp_compact"), out)]
        assert st[0] == st[1] == 0
        for part in (slice(0, 14), slice(14, 16)):
            assert np.max(np.abs(out[0][part] - out[1][part])) <= RTOL_FP64 * np.max(np.abs(out[0]))


def test_integer_pipe_conversions(lib):
    rng = np.random.default_rng(5)
    x = np.concatenate([rng.standard_normal(200) * 10.0 ** rng.uniform(-30, 30, 200),
                        [0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, 1e39, -1e39, 1e-39]])
    for v in x:
        f = lib.c64_to_f32(v)
        if 1.2e-38 < abs(v) < 3.4e38:
            assert abs(f - v) <= 2.0 ** -23 * abs(v) and abs(f) <= abs(v)  # truncated
        else:
            assert f == (0.0 if abs(v) < 1e-38 else np.copysign(np.inf, v))
        if abs(f) > 1.2e-38 or f == 0.0:
            assert lib.c64_to_f64(f) == f
    assert np.isnan(lib.c64_to_f32(np.nan)) and np.isnan(lib.c64_to_f64(np.nan))


def test_integer_products_are_the_hardware_s(lib):
    """soft_mul64 against the FP64 product, bit for bit: random significands, short ones
    (ties), zeros of both signs and exponents over the range; beyond it the products are
    flagged, and infinities and NaN too."""
    lib.c64_soft_mul.restype = ctypes.c_double
    lib.c64_soft_mul.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.POINTER(ctypes.c_int)]
    rng = np.random.default_rng(11)
    x, y = rng.uniform(-2, 2, 40000), rng.uniform(-2, 2, 40000)
    x[::5] = rng.integers(-(1 << 27), 1 << 27, x[::5].size) * 2.0 ** -20
    y[::5] = rng.integers(-(1 << 27), 1 << 27, x[::5].size) * 2.0 ** -25
    x[1::5] *= 2.0 ** rng.integers(-400, 400, x[1::5].size)
    y[1::5] *= 2.0 ** rng.integers(-80, 80, x[1::5].size)
    x[2::50], y[3::50], x[4::50] = 0.0, -0.0, 1.0
    ok = ctypes.c_int()
    for a, b in zip(x.tolist(), y.tolist()):
        r = lib.c64_soft_mul(a, b, ctypes.byref(ok))
        assert ok.value and np.float64(r).tobytes() == np.float64(a * b).tobytes(), (a, b, r)
    for a, b in ((1e-200, 1e-200), (1e200, 1e200), (np.inf, 2.0), (3.0, np.nan), (-np.inf, -np.inf), (np.nan, np.nan)):
        lib.c64_soft_mul(a, b, ctypes.byref(ok))
        assert not ok.value, (a, b)


@pytest.mark.parametrize("ep", EOS)
def test_integer_products_leave_the_forms_as_they_are(lib, orc, ep):
    """Flux, speed and status bit for bit those of the hardware's products, in ordinary
    states and where products leave the range (tiny and large momenta, NaN, infinities)."""
    rng = np.random.default_rng(5)
    for q in phase_states(orc, ep, rng, 40, (1.0, 0.3, 1e-6), 0.1):
        for v, x in ((None, 0), (3, 0.0), (3, 1e-170), (4, 1e-300), (2, 1e160), (5, np.inf), (7, np.nan), (10, -np.inf),
                     (6, -q[6]), (4, np.nan)):
            p = q.copy()
            if v is not None:
                p[v] = x
            s0, a = ev(lib, "c64_plain", ep, p)
            s1, b = ev(lib, "c64_compact", ep, p)
            assert s0 == s1 and a.tobytes() == b.tobytes(), (v, x)


@pytest.mark.parametrize("ep", EOS)
def test_integer_products_leave_the_vjp_as_it_is(lib, orc, ep):
    """As above for the adjoint's cell."""
    dp = ctypes.POINTER(ctypes.c_double)
    rng = np.random.default_rng(6)
    e = np.array(ep, dtype=np.float64)
    for s in phase_states(orc, ep, rng, 30, (1.0,), 0.1):
        fb, lb = rng.standard_normal(14), rng.standard_normal()
        for v, x in ((None, 0), (2, 0.0), (3, 1e-170), (1, 1e160), (4, np.inf), (6, np.nan)):
            q, out = s[1:].copy(), [np.zeros(16), np.zeros(16)]
            if v is not None:
                q[v] = x
            st = []
            for n, o in zip(("c64_vjp_plain", "c64_vjp_compact"), out):
                o[:14] = fb
                st.append(getattr(lib, n)(e.ctypes.data_as(dp), q.ctypes.data_as(dp), fb.ctypes.data_as(dp),
                                          ctypes.c_double(lb), o.ctypes.data_as(dp)))
            assert st[0] == st[1] and out[0].tobytes() == out[1].tobytes(), (v, x)
