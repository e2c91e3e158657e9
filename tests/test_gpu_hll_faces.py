"""The HLL face evaluator on more faces than one thread block holds (GPU)."""
import numpy as np
import pytest

from helpers import RTOL_FP64, assert_within_sensitivity, ulp_sensitivity
from test_gpu_mph import eos_pair, oracle_pb, random_mph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 65, 200])
@pytest.mark.parametrize("own_speeds", [True, False])
def test_hll_every_face(hyp, orc, n, own_speeds):
    """Every face of an n-face array matches the oracle (the tolerance of test_twophase_evaluators)."""
    from hyperelasticsolver_gb300 import NumFluxes as NF
    Q = random_mph(orc, n + 1, np.random.default_rng(17))
    pb, l, r = oracle_pb(orc), Q[:-1], Q[1:]
    el, er = orc.speeds(pb, l), orc.speeds(pb, r)
    if not own_speeds:
        el, er = 1.1 * el, 1.2 * er
    _, dm, dp = NF.hll(eos_pair(hyp), l, r, None if own_speeds else [el, er])
    ref = orc.hll(pb, l, r, el, er)
    for k, got in enumerate((dm, dp)):
        sens = ulp_sensitivity(lambda a, b: orc.hll(pb, a, b, el, er)[k], (l, r), trials=2)
        assert_within_sensitivity(got, ref[k], sens, RTOL_FP64, f"hll D{'-+'[k]}", axis=0)


@pytest.mark.parametrize("n", [1, 64, 65, 200])
@pytest.mark.parametrize("general", [False, True])
def test_lxf_every_face(hyp, orc, n, general):
    """The two-phase LxF face evaluator, on a block's edges and with main.jl:133's general
    exponents (the tolerance of test_twophase_evaluators)."""
    from hyperelasticsolver_gb300 import NumFluxes as NF
    from test_gpu_two_faces import setup
    eos, pb = setup(hyp, orc, 3, "lxf", general)
    rng = np.random.default_rng(23)
    Q = random_mph(orc, n + 1, rng)
    l, r, lam = Q[:-1], Q[1:], rng.uniform(5.0, 8.0, n)
    got, ref = NF.lxf(eos, l, r, lam), orc.lxf(pb, l, r, lam)
    for k, what in enumerate(("cons", "D-", "D+")):
        sens = ulp_sensitivity(lambda a, b: orc.lxf(pb, a, b, lam)[k], (l, r), trials=2)
        assert_within_sensitivity(got[k], ref[k], sens, RTOL_FP64, f"lxf {what}", axis=0)
