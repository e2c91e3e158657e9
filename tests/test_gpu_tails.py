"""Long FP64 runs, in which every front has drawn a tail down to the smallest numbers behind
(ahead of) it: on grids large enough for the integer products (hyp_cell64.cuh) the same bits
as on small ones, and the same time a step as a short run (GPU)."""
import numpy as np
import pytest

from hyperelasticsolver_gb300 import _cases as C
from test_gpu_mph import B0_SOFT

pytestmark = pytest.mark.gpu


def ends(hyp, eos):
    """Strained on the left, no strain on the right: shears that are zero there, with tails."""
    return [hyp.Hyperelasticity.prim2cons(eos, p) for p in C.adjoint_states(eos)]


@pytest.mark.parametrize("flux,K", [("rusanov", 600), ("lxf", 1100)])  # an LxF front halves its tail a cell
def test_single_phase_same_bits(hyp, flux, K):
    """16384 cells in one launch with the hardware's products, the middle of 32768 of the same
    size, and the problems of a batch of 1040 tiles."""
    eos, n = hyp.Barton2009(), 16384
    ql, qr = ends(hyp, eos)
    out = []
    for w in (1, 2):
        with hyp.Solver(eos, w * n, flux=flux, X=float(w)) as s:
            s.init_riemann(ql, qr)
            s.step(max_steps=K)
            out.append((s.time(), s.download()))
    (t, a), (tw, b) = out
    assert 0 < np.min(np.abs(a[a != 0])) < 1e-300  # there are tails
    assert t == tw and np.array_equal(b[:, n // 2:n // 2 + n], a)
    assert np.all(b[:, :n // 2] == b[:, :1]) and np.all(b[:, -(n // 2):] == b[:, -1:])
    with hyp.Batch(eos, [n] * 8, flux=flux, precision="fp64") as s:
        s.upload(np.tile(C.initial_condition(ql, qr, n), (1, 8)))
        s.step(K)
        q = s.download()
        assert all(np.array_equal(s.problem(q, p), a) for p in range(8)) and np.all(s.status()[0] == t[0])


@pytest.mark.parametrize("flux", ["hll", "lxf"])
def test_two_phase_same_bits(hyp, flux):
    """4096 cells against the middle of 16384: there all cell, face and update kernels take the
    integer products, and the LxF faces keep marks, of which a few blocks' are set."""
    from hyperelasticsolver_gb300 import HyperelasticityMPh as HM
    eos = (hyp.Barton2009(), hyp.Barton2009(_b0=B0_SOFT))
    Ql, Qr = HM.initial_states(eos, 6)
    n, K, out = 4096, 300, []
    for w in (1, 4):
        with hyp.Solver(eos, w * n, model="multi", flux=flux, X=float(w)) as s:
            s.init_riemann(Ql, Qr)
            s.step(max_steps=K)
            out.append((s.time(), s.download()))
    (t, a), (tw, b) = out
    lo = 3 * n // 2
    assert t == tw and np.array_equal(b[:, lo:lo + n], a)
    assert np.all(b[:, :lo] == b[:, :1]) and np.all(b[:, -lo:] == b[:, -1:])


def test_adjoint_same_values_and_rate(hyp):
    """The reverse pass over 600 steps: 16384 cells (the hardware's products) against the middle
    of 65536, to the order of a sum over blocks; and a step of
    it as fast as one of 50, here and forward."""
    eos, n, K, w = hyp.Barton2009(), 16384, 600, 4
    ql, qr = ends(hyp, eos)
    seed = np.random.default_rng(7).standard_normal((14, n))
    seed[:, :n // 4] = seed[:, -n // 4:] = 0.0  # nothing of it reaches an end in 600 steps
    with hyp.Solver(eos, n) as s:
        s.init_riemann(ql, qr)
        s.record(K, 50)
        g, ge = s.adjoint(seed)
    lo = (w - 1) * n // 2
    wide = np.zeros((14, w * n))
    wide[:, lo:lo + n] = seed
    with hyp.Solver(eos, w * n, X=float(w)) as s:
        s.init_riemann(ql, qr)
        s.record(K, 50)
        h, he = s.adjoint(wide)
        assert np.max(np.abs(h[:, lo:lo + n] - g)) <= 1e-12 * np.max(np.abs(g))
        assert np.max(np.abs(he - ge)) <= 1e-12 * np.max(np.abs(ge))
        us = {}
        dense = np.random.default_rng(8).standard_normal((14, w * n))
        for k in (50, K):
            s.init_riemann(ql, qr)
            s.record(k, 50)
            runs = []
            for _ in range(3):
                s.adjoint(dense)
                runs.append(s.adjoint_timing())
            us[k] = [1e3 * min(r[m] for r in runs) / k for m in ("ms_recompute", "ms_adjoint")]
        print("us a step, forward and reverse:", us)
        assert us[K][0] <= 1.25 * us[50][0] and us[K][1] <= 1.25 * us[50][1]
