"""The FP64 forms' integer products (hyp_cell64.cuh, host build) where their range ends: the
tail of a wave, subnormal and non-finite values. The same bits as the hardware's products,
and no detour by the general forms. CPU only."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
EP = np.array((8.93, 4.6, 3.9e-4, 300, 2.1, 1, 3, 2), dtype=np.float64)
DP = ctypes.POINTER(ctypes.c_double)
DONE, PLAIN, GENERAL = 0, 1, 2


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(tempfile.mkdtemp(prefix="hyp_t64_"), "t64.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                        os.path.join(HERE, "tails64_shim.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)


def cell(lib, q):
    out, plain, st, q = np.zeros(16), np.zeros(16), (ctypes.c_int * 2)(), np.ascontiguousarray(q)
    held = lib.t64_cell(EP.ctypes.data_as(DP), q.ctypes.data_as(DP), out.ctypes.data_as(DP), plain.ctypes.data_as(DP), st)
    return held, out, plain, tuple(st)


def vjp(lib, q, fb, lb):
    left = (ctypes.c_int * 2)()
    out, plain = np.zeros(16), np.zeros(16)
    out[:14] = plain[:14] = fb
    q, fb = np.ascontiguousarray(q), np.ascontiguousarray(fb)
    lib.t64_vjp(EP.ctypes.data_as(DP), q.ctypes.data_as(DP), fb.ctypes.data_as(DP), ctypes.c_double(lb),
                out.ctypes.data_as(DP), plain.ctypes.data_as(DP), left)
    return tuple(left), out, plain


def tail(rng, t, alpha=1.0):
    """A phase at rest but for velocities, shears and an entropy part of size t."""
    rho = alpha * 8.93
    F = np.eye(3) + t * rng.standard_normal((3, 3))
    return np.concatenate([[alpha, rho], rho * t * rng.standard_normal(3), [rho * t * abs(rng.standard_normal())],
                           rho * F.reshape(-1, order="F")])


@pytest.mark.parametrize("alpha", [1.0, 0.3])
def test_wave_tails(lib, alpha):
    """Disturbances of 1e-1 down to the last subnormal number: bit for bit the hardware's
    products; the integer ones down to 1e-70, where their fourth powers are still in range."""
    rng = np.random.default_rng(3)
    for k in range(1, 325):
        q = tail(rng, 10.0 ** -k if k < 324 else 5e-324, alpha)
        held, a, b, st = cell(lib, q)
        assert a.tobytes() == b.tobytes() and st == (0, 0), k
        assert held or k > 70, k


def test_wave_tails_of_the_adjoint(lib):
    """The same for the reverse cell, with adjoints of ordinary size and with a tail of their
    own: what the integer products leave, the hardware's do, and never the general form."""
    rng = np.random.default_rng(4)
    for k in range(1, 325):
        q = tail(rng, 10.0 ** -k if k < 324 else 5e-324)[1:]
        for size in (1.0, 10.0 ** -k):
            fb, lb = size * rng.standard_normal(14), size * rng.standard_normal()
            left, a, b = vjp(lib, q, fb, lb)
            assert a.tobytes() == b.tobytes(), (k, size)
            assert left[0] in (DONE, PLAIN) and left[1] == DONE, (k, size)
            assert left[0] == DONE or k > 40, (k, size)


@pytest.mark.parametrize("x", [5e-324, 1e-310, -2e-308, 1e-170, 1e160, 1e300, np.inf, -np.inf, np.nan])
def test_values_past_the_range(lib, x):
    """Every entry of a cell in turn subnormal, tiny, huge, infinite or NaN, beside zeros and
    ordinary values: the hardware's bits and status."""
    rng = np.random.default_rng(5)
    for base in (tail(rng, 0.05, 0.4), tail(rng, 0.0, 0.4)):
        for v in range(15):
            q = base.copy()
            q[v] = x
            held, a, b, st = cell(lib, q)
            assert st[0] == st[1] and a.tobytes() == b.tobytes(), v
            if v:
                fb = rng.standard_normal(14)
                for f in (fb, np.where(np.arange(14) % 3, fb, 0.0), np.where(np.arange(14) == 4, x, fb)):
                    left, a, b = vjp(lib, q[1:], f, 0.3)
                    assert a.tobytes() == b.tobytes(), v


@pytest.mark.parametrize("lxf", [False, True])
def test_step_scalars(lib, lxf):
    """dt = cfl dx / max speed, lambda and dt/dx against divisions: 2 ulps a quotient where all
    of them are ordinary, and the divisions themselves (infinities and zeros included) where
    an argument or a quotient leaves the range of the reciprocals."""
    rng = np.random.default_rng(6)
    cases = [(0.5, 10.0 ** a, 10.0 ** b) for a, b in rng.uniform(-8, 8, (200, 2))]
    cases += [(0.5, 10.0 ** a, 10.0 ** b) for a, b in rng.uniform(-320, 308, (2000, 2))]
    cases += [(0.5, x, y) for x in (1e-240, 1e-3, 1e240) for y in (0.0, 5e-324, 1e-247, 1e-100, 1.0, 1e100, 1e246, 1e300, np.inf)]
    fast = 0
    for cfl, dx, lmax in cases:
        out = np.zeros(3)
        lib.t64_scalars(ctypes.c_double(cfl), ctypes.c_double(dx), ctypes.c_double(lmax), int(lxf), out.ctypes.data_as(DP))
        with np.errstate(all="ignore"):
            dt = np.float64(cfl) * dx / np.float64(lmax)
            lam = dx / dt
            ref = np.array([dt, lam, np.float64(1.0) / lam if lxf else dt / dx])
        if not lxf:
            out[1] = ref[1]  # not a Rusanov step's
        assert np.array_equal(np.isnan(out), np.isnan(ref)), (dx, lmax, out, ref)
        fin = np.isfinite(ref) & (np.abs(ref) > 1e-290)
        assert np.all(np.abs(out[fin] - ref[fin]) <= 6 * 2.0 ** -53 * ref[fin]), (dx, lmax, out, ref)
        assert np.array_equal(out[~fin], ref[~fin], equal_nan=True), (dx, lmax, out, ref)
        fast += bool(fin.all())
    assert fast > 300
