"""The step's path integrals (hyp_paths64.cuh, host build): the number of nodes taken and
the value, against all six nodes of the general forms. CPU only."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
DEFAULT = [(8.93, 4.6, 3.9e-4, 300, 2.1, 1, 3, 2), (8.93, 4.6, 3.9e-4, 300, 2.1 * 0.1 ** 0.5, 1, 3, 2)]
GENERAL = [(8.93, 6.22, 9.0e-4, 300, 3.16, 1, 3.577, 2.088), (8.93, 6.22, 9.0e-4, 300, 1.0, 1, 3.577, 2.088)]
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(tempfile.mkdtemp(prefix="hyp_p64_"), "p64.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                        os.path.join(HERE, "paths64_shim.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)


def path(lib, eos, a, b):
    x, w = np.polynomial.legendre.leggauss(6)
    dp = ctypes.POINTER(ctypes.c_double)
    arr = [np.ascontiguousarray(v, dtype=np.float64) for v in
           (np.concatenate(eos), np.concatenate([0.5 * (x + 1), 0.5 * w]), a, b, np.zeros(30), np.zeros(30))]
    n = lib.p64_path(*[v.ctypes.data_as(dp) for v in arr])
    return n, arr[4], arr[5]


def state(orc, eos, rng, a1, near=None, size=0.0):
    """A two-phase state; `near` a primitive one that it differs from by about `size`."""
    P = np.empty(30)
    for p in range(2):
        F = np.eye(3) + 0.03 * rng.standard_normal((3, 3))
        P[15 * p:15 * p + 15] = [a1 if p == 0 else 1 - a1, 8.93 / np.linalg.det(F), *rng.uniform(-0.4, 0.4, 3),
                                 rng.uniform(0, 5e-4), *F.reshape(-1, order="F")]
    if near is not None:
        keep = P[[0, 15]].copy()
        P = near + size * (P - near)
        P[[0, 15]] = near[[0, 15]] + size * (keep - near[[0, 15]])
        P[15] = 1 - P[0]
    pb = orc.problem(model=orc.MODEL_MULTI, flux=orc.FLUX_HLL, eos=tuple(orc.barton2009(*e) for e in eos))
    return P, np.asarray(orc.prim2cons(pb, P)).reshape(-1)


@pytest.mark.parametrize("eos", [DEFAULT, GENERAL])
@pytest.mark.parametrize("a1", [0.5, 0.03, 1e-6])
@pytest.mark.parametrize("size", [1e-7, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 0.1, 1.0])
def test_value_to_rounding(lib, orc, eos, a1, size):
    """Whatever the number of nodes, each phase's rows agree with the six-node value to the
    rounding of both evaluations: a node's B carries a few hundred operations, so 1000 eps
    of B d(alpha) on the scale of the largest row, plus the rule's own share, eps/16 of
    alpha B. All node counts occur over the sizes."""
    rng = np.random.default_rng(31)
    for _ in range(12):
        P, a = state(orc, eos, rng, a1)
        _, b = state(orc, eos, rng, min(1.7 * a1, 0.8), near=P, size=size)
        n, acc, ref = path(lib, eos, a, b)
        assert n in (2, 3, 6)
        if size >= 0.1:
            assert n == 6  # far from smooth
        if size <= 1e-7:
            assert n == 2
        for p in range(2):
            r = slice(15 * p, 15 * p + 15)
            da = abs(b[15 * p] - a[15 * p])
            big = np.max(np.abs(ref[r])) / da  # B's scale
            assert np.max(np.abs(acc[r] - ref[r])) <= big * (1000 * EPS * da + EPS / 16 * min(a[15 * p], b[15 * p]))


def test_unsafe_paths_take_all_nodes(lib, orc):
    """NaN, a non-positive fraction or determinant, a state at the entropy clamp and equal
    fractions with a large strain jump (no integral, but its nodes' statuses count)."""
    rng = np.random.default_rng(5)
    P, a = state(orc, DEFAULT, rng, 0.4)
    _, b = state(orc, DEFAULT, rng, 0.41, near=P, size=1e-6)
    assert path(lib, DEFAULT, a, b)[0] == 2
    for j, v in ((0, np.nan), (0, -0.1), (0, 0.0), (6, np.nan), (21, -5.0), (2, np.inf), (5, np.nan), (20, -40.0)):
        for side in range(2):
            q = [a.copy(), b.copy()]
            q[side][j] = v
            assert path(lib, DEFAULT, *q)[0] == 6
    c = a.copy()
    c[6:15] = -c[6:15]
    assert path(lib, DEFAULT, a, c)[0] == 6
