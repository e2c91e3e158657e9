"""The two-phase LxF face evaluator between close states: D- and D+ are the path integral by
itself, right relative to its own size however small the volume fractions' jump (GPU)."""
import numpy as np
import pytest

from helpers import RTOL_FP64
from test_gpu_two_faces import setup, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("jump", [1e-4, 1e-6, 1e-8, 1e-10])
def test_fluctuations_of_close_states(hyp, orc, general, jump):
    """Against the oracle, each phase's rows at the parity tolerance of the face's largest one;
    the fractions' difference is exact, so the tolerance is that of B."""
    from hyperelasticsolver_gb300 import NumFluxes as NF
    eos, pb = setup(hyp, orc, 3, "lxf", general)
    n = 200
    rng = np.random.default_rng(8)
    P = np.asarray(orc.cons2prim(pb, np.ascontiguousarray(smooth_state(orc, pb, n, True).T)))
    R = P.copy()
    R[:, 0] *= 1 + jump
    R[:, 15] = 1 - R[:, 0]
    for p in (0, 15):
        R[:, p + 2:p + 5] += rng.choice([0.003, 0.01, 0.03], (n, 1)) * rng.standard_normal((n, 3))
        R[:, p + 5] = P[:, p + 5] = rng.choice([2e-4, 3e-3], n)  # cold and hot
    l, r = (np.asarray(orc.prim2cons(pb, x)) for x in (P, R))
    _, dm, dp = NF.lxf(eos, l, r, np.full(n, 6.0))
    _, om, op = orc.lxf(pb, l, r, np.full(n, 6.0))
    for got, ref in ((dm, om), (dp, op)):
        for p in (0, 15):
            big = np.max(np.abs(ref[:, p:p + 15]), axis=1)
            err = np.max(np.abs(got[:, p:p + 15] - ref[:, p:p + 15]), axis=1) / big
            print(f"jump {jump:.0e} phase {p // 15}: {err.max():.1e}")
            assert np.all(big > 0) and np.all(err <= RTOL_FP64)
