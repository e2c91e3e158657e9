"""The nodes of the step's path integrals (hyp_paths64.cuh, host build) where the volume
fractions jump by far less than the states. CPU only."""
import numpy as np
import pytest

from test_paths64_host import DEFAULT, EPS, GENERAL, lib, path, state  # noqa: F401 (lib: a fixture)


@pytest.mark.parametrize("eos", [DEFAULT, GENERAL])
@pytest.mark.parametrize("jump", [1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-12])
@pytest.mark.parametrize("du,dF", [(0.01, 0.0), (0.03, 1e-3), (0.1, 0.0), (0.0, 0.01), (0.1, 0.02)])
def test_small_fraction_jumps(lib, orc, eos, jump, du, dF):  # noqa: F811
    """The bound of test_paths64_host.test_value_to_rounding, for fractions whose relative jump
    is 1e-6 to 1e-12 and velocities and distortions that jump on their own."""
    rng = np.random.default_rng(17)
    pb = orc.problem(model=orc.MODEL_MULTI, flux=orc.FLUX_HLL, eos=tuple(orc.barton2009(*e) for e in eos))
    for _ in range(40):
        P, a = state(orc, eos, rng, 0.4)
        R = P.copy()
        R[0] = 0.4 * (1 + jump)
        R[15] = 1 - R[0]
        for p in (0, 15):
            R[p + 2:p + 5] += du * rng.standard_normal(3)
            R[p + 6:p + 15] += dF * rng.standard_normal(9)
            R[p + 1] = 8.93 / np.linalg.det(R[p + 6:p + 15].reshape(3, 3))
        b = np.asarray(orc.prim2cons(pb, R)).reshape(-1)
        _, acc, ref = path(lib, eos, a, b)
        for p in (0, 15):
            r = slice(p, p + 15)
            da = abs(b[p] - a[p])
            big = np.max(np.abs(ref[r])) / da  # B's scale
            assert np.max(np.abs(acc[r] - ref[r])) <= big * (1000 * EPS * da + EPS / 16 * min(a[p], b[p]))
