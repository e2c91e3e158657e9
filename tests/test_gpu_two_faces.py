"""The three routes of a two-phase FP64 face (volume fractions equal: no path integral;
a few listed faces: 16 lanes each; many: a thread each) against the oracle (GPU)."""
import numpy as np
import pytest

from helpers import RTOL_FP64, assert_close_soa
from test_gpu_mph import B0_SOFT

pytestmark = pytest.mark.gpu

GENERAL = dict(c0=6.22, cv=9.0e-4, b0=3.16, beta=3.577, gamma=2.088)  # main.jl:133's exponents


def setup(hyp, orc, nx, flux, general=False, bc=0):
    two = (dict(GENERAL), dict(GENERAL, b0=3.16 * 0.1 ** 0.5)) if general else (dict(), dict(b0=B0_SOFT))
    eos = tuple(hyp.Barton2009(**{"_" + k: v for k, v in d.items()}) for d in two)
    pb = orc.problem(model=orc.MODEL_MULTI, flux=orc.FLUX_HLL if flux == "hll" else orc.FLUX_LXF, nx=nx, cfl=0.5,
                     bc=bc, eos=tuple(orc.barton2009(**d) for d in two))
    return eos, pb


def smooth_state(orc, pb, nx, alpha_varies, seed=6):
    """Strain, velocity, entropy and (where it varies) volume fraction as slow waves."""
    rng = np.random.default_rng(seed)
    x = (np.arange(nx) + 0.5) / nx
    wave = lambda amp, k=3: amp * np.sin(2 * np.pi * (k * x + rng.uniform()))
    a1 = 0.4 + (wave(0.2) if alpha_varies else 0.0 * x)
    P = np.empty((nx, 30))
    for p in range(2):
        F = np.eye(3)[None] + np.stack([wave(0.02) for _ in range(9)], -1).reshape(nx, 3, 3)
        P[:, 15 * p] = a1 if p == 0 else 1.0 - a1
        P[:, 15 * p + 1] = 8.93 / np.linalg.det(F)
        P[:, 15 * p + 2:15 * p + 5] = np.stack([wave(0.3) for _ in range(3)], -1)
        P[:, 15 * p + 5] = 2e-4 + wave(1e-4)
        P[:, 15 * p + 6:15 * p + 15] = F.transpose(0, 2, 1).reshape(nx, 9)
    return np.ascontiguousarray(orc.prim2cons(pb, P).T)


# 3 and 65: the ends and a block's edge; 1000: lists done by groups; 12300 listed faces
# (above 80 a multiprocessor on 152 of them): a thread each
@pytest.mark.parametrize("flux", ["hll", "lxf"])
@pytest.mark.parametrize("nx,steps", [(3, 4), (65, 4), (1000, 2), (12300, 1)])
@pytest.mark.parametrize("alpha_varies", [True, False])
def test_routes_match_oracle(hyp, orc, flux, nx, steps, alpha_varies):
    eos, pb = setup(hyp, orc, nx, flux, bc=orc.BC_TRANSMISSIVE)
    Q0 = smooth_state(orc, pb, nx, alpha_varies)
    Qo, so, to, _ = orc.run(pb, Q0, max_steps=steps)
    with hyp.Solver(eos, nx, model="multi", flux=flux, bc="transmissive") as s:
        s.upload(Q0)
        n, t = s.step(max_steps=steps)
        assert n == steps and abs(t - to) <= RTOL_FP64 * to
        assert_close_soa(s.download(), Qo, RTOL_FP64, f"{flux} {nx}")


@pytest.mark.parametrize("flux", ["hll", "lxf"])
@pytest.mark.parametrize("alpha_varies", [True, False])
def test_general_exponents(hyp, orc, flux, alpha_varies):
    eos, pb = setup(hyp, orc, 200, flux, general=True)
    Q0 = smooth_state(orc, pb, 200, alpha_varies)
    Qo, so, to, _ = orc.run(pb, Q0, max_steps=3)
    with hyp.Solver(eos, 200, model="multi", flux=flux) as s:
        s.upload(Q0)
        n, t = s.step(max_steps=3)
        assert abs(t - to) <= RTOL_FP64 * to
        assert_close_soa(s.download(), Qo, RTOL_FP64, flux)


@pytest.mark.parametrize("flux", ["hll", "lxf"])
def test_strong_strain_jump_takes_the_integrals(hyp, orc, flux):
    """Equal volume fractions but a strain jump too large to rule out a singular state on
    the way: the face is listed and matches the oracle."""
    eos, pb = setup(hyp, orc, 40, flux)
    c, s_ = np.cos(0.9), np.sin(0.9)
    P = smooth_state(orc, pb, 40, False)
    prims = orc.cons2prim(pb, np.ascontiguousarray(P.T))
    for p in range(2):
        A = prims[20:, 15 * p + 6:15 * p + 15].reshape(-1, 3, 3).transpose(0, 2, 1)
        A = np.array([[1, 0, 0], [0, c, -s_], [0, s_, c]]) @ A
        prims[20:, 15 * p + 6:15 * p + 15] = A.transpose(0, 2, 1).reshape(-1, 9)
    Q0 = np.ascontiguousarray(orc.prim2cons(pb, prims).T)
    Qo, so, to, _ = orc.run(pb, Q0, max_steps=1)
    with hyp.Solver(eos, 40, model="multi", flux=flux) as s:
        s.upload(Q0)
        s.step(max_steps=1)
        assert_close_soa(s.download(), Qo, RTOL_FP64, flux)


@pytest.mark.parametrize("flux", ["hll", "lxf"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_singular_state_on_the_path_is_refused(hyp, orc, flux, precision):
    """Two admissible cells of equal volume fractions whose distortions differ by a half
    turn: det of the path's middle is not positive, and the step says so."""
    eos, pb = setup(hyp, orc, 40, flux)
    P = np.zeros((40, 30))
    for p in range(2):
        P[:, 15 * p], P[:, 15 * p + 1] = 0.5, 8.93
        A = np.tile(np.eye(3), (40, 1, 1))
        A[20:] = np.diag([1.0, -1.0, -1.0])
        P[:, 15 * p + 6:15 * p + 15] = A.reshape(40, 9)
    Q0 = np.ascontiguousarray(orc.prim2cons(pb, P).T)
    with hyp.Solver(eos, 40, model="multi", flux=flux, precision=precision) as s:
        s.upload(Q0)
        with pytest.raises(hyp._lib.NegativeDeterminantError):
            s.step(max_steps=2)
