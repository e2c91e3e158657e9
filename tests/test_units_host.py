"""The FP64 forms do not depend on the system of units (hyp_cell64.cuh, hyp_physics.cuh, host
build). A power of two in the unit of velocity or of density scales every operation exactly,
so the results are compared bit for bit. CPU only."""
import ctypes

import numpy as np
import pytest

from test_cell64_host import EOS, ev, lib, phase_states  # noqa: F401 (lib: the module's fixture)

# 2^-23 and 2^-30: speeds of 5e-7 and 4e-9 (cm/ps and below); 2^10 and 2^20: m/s and mm/s
SPEEDS = [-40, -30, -23, -12, 10, 20, 30, 45]


def in_units(ep, q, ku, kr):
    """EOS and one phase (15 values) with velocities times 2^ku and densities times 2^kr."""
    u, r = 2.0 ** ku, 2.0 ** kr
    rho0, c0, cv, t0, b0, *rest = ep
    p = q.copy()
    p[1:] *= r
    p[2:5] *= u
    p[5] *= u * u
    return (rho0 * r, c0 * u, cv * u * u, t0, b0 * u, *rest), p


def out_units(out, ku, kr):
    u, r = 2.0 ** ku, 2.0 ** kr
    s = np.empty(16)
    s[0], s[1:4], s[4], s[5:14], s[14:] = r * u, r * u * u, r * u ** 3, r * u, u
    return out * s


@pytest.mark.parametrize("ep", EOS)
@pytest.mark.parametrize("strain", [0.0, 0.05, 0.1, 0.3])
def test_general_forms(lib, orc, ep, strain):  # noqa: F811
    """hyp_physics.cuh: the function-level evaluators' forms and the step's for close speeds."""
    rng = np.random.default_rng(13)
    for q in phase_states(orc, ep, rng, 30, (1.0, 0.25), strain):
        st, ref = ev(lib, "c64_general", ep, q)
        assert st == 0
        for ku in SPEEDS:
            for kr in (-40, 0, 10):
                s, out = ev(lib, "c64_general", *in_units(ep, q, ku, kr))
                assert s == 0 and np.array_equal(out, out_units(ref, ku, kr)), (ku, kr)


@pytest.mark.parametrize("ep", EOS)
@pytest.mark.parametrize("strain", [0.0, 0.02, 0.1, 0.3])
@pytest.mark.parametrize("form", ["c64_compact", "c64_plain"])
def test_compact_forms(lib, orc, ep, strain, form):  # noqa: F811
    rng = np.random.default_rng(12)
    for q in phase_states(orc, ep, rng, 20, (1.0, 0.25), strain):
        st, ref = ev(lib, form, ep, q)
        assert st == 0
        for ku in SPEEDS:
            for kr in (-40, 0, 10):
                s, out = ev(lib, form, *in_units(ep, q, ku, kr))
                assert s == 0 and np.array_equal(out, out_units(ref, ku, kr)), (ku, kr)
