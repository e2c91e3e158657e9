"""A run of FP64 steps does not depend on how it is cut into calls: steps inside one call
share kernels (update and next cell pass in one), the first and last of a call do not
(GPU). Bitwise: the same arithmetic either way."""
import numpy as np
import pytest

from hyperelasticsolver_gb300 import _cases as C

pytestmark = pytest.mark.gpu

CUTS = [[1] * 27, [27], [2, 13, 12], [12, 15], [26, 1]]  # 12 steps are one captured graph


def state(hyp, n, seed=3):
    eos = hyp.Barton2009()
    return eos, C.segment_fill(hyp.Hyperelasticity.prim2cons(eos, C.segment_states(eos, 8, seed=seed)), n)


@pytest.mark.parametrize("n", [3, 63, 64, 127, 128, 300, 9576, 9577, 19304, 19305])  # 9576, 19304: the last of each form of one launch on 152 SMs
@pytest.mark.parametrize("flux,bc", [("rusanov", "frozen"), ("lxf", "transmissive")])
def test_cuts_agree(hyp, n, flux, bc):
    eos, Q0 = state(hyp, n)
    out = []
    for cut in CUTS:
        with hyp.Solver(eos, n, flux=flux, bc=bc) as s:
            s.upload(Q0)
            for k in cut:
                assert s.step(max_steps=k)[0] == k
            out.append((s.download(), s.time()))
    for Q, t in out[1:]:
        assert np.array_equal(Q, out[0][0]) and t == out[0][1]


def test_stop_at_t_end_and_go_on(hyp):
    """Steps past t_end leave everything as it is; the run then goes on as if never stopped;
    profiled, time-logged and recorded runs take the same steps."""
    eos, Q0 = state(hyp, 200)
    ref = []
    with hyp.Solver(eos, 200) as s:
        s.upload(Q0)
        for _ in range(31):
            ref.append((s.step(max_steps=1)[1], s.download()))
    for stop in (1, 2, 3, 12, 14):
        with hyp.Solver(eos, 200) as s:
            s.upload(Q0)
            t_end = 0.5 * (ref[stop - 2][0] + ref[stop - 1][0]) if stop > 1 else 0.5 * ref[0][0]
            assert s.step(t_end=t_end) == (stop, ref[stop - 1][0])
            assert np.array_equal(s.download(), ref[stop - 1][1])
            assert s.step(max_steps=40, t_end=t_end)[0] == 0
            s.set_profiling(True)
            s.step(max_steps=3)
            s.set_profiling(False)
            th, _ = s.step_times(5)
            assert np.array_equal(th, [ref[stop + 3 + k][0] for k in range(5)])
            s.record(31 - stop - 8, 4)
            assert s.time()[0] == ref[30][0] and np.array_equal(s.download(), ref[30][1])


def test_batch_cuts_agree(hyp):
    eos = hyp.Barton2009()
    sizes = [3, 127, 128, 500]
    Q0 = np.concatenate([state(hyp, n, seed=k)[1] for k, n in enumerate(sizes)], axis=1)
    out = []
    for cut in ([1] * 9, [9], [4, 5]):
        with hyp.Batch(eos, sizes, precision="fp64") as b:
            b.upload(Q0)
            for k in cut:
                b.step(k)
            mid = b.status()[0][3] + 1e-9  # the largest problem stops at once, coarser ones when they pass it
            b.step(5, t_end=mid)
            b.step(3)
            out.append((b.download(), *b.status()))
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))
    Q, t, steps = out[0]
    for p, n in enumerate(sizes):  # each problem as a single run of its own
        with hyp.Solver(eos, n) as s:
            lo = sum(sizes[:p])
            s.upload(np.ascontiguousarray(Q0[:, lo:lo + n]))
            _, tp = s.step(max_steps=int(steps[p]))
            assert tp == t[p] and np.array_equal(s.download(), Q[:, lo:lo + n])


@pytest.mark.parametrize("n", [3, 64, 65, 300])
@pytest.mark.parametrize("flux", ["hll", "lxf"])
@pytest.mark.parametrize("relax", [None, "mechanical"])
def test_two_phase_cuts_agree(hyp, n, flux, relax):
    from hyperelasticsolver_gb300 import HyperelasticityMPh as HM
    eos = (hyp.Barton2009(), hyp.Barton2009(_b0=2.1 * 0.1 ** 0.5))
    Ql, Qr = HM.initial_states(eos, 4)
    out = []
    for cut in CUTS:
        with hyp.Solver(eos, n, model="multi", flux=flux, relax=relax) as s:
            s.init_tanh(Ql, Qr, 0.2)
            for k in cut:
                assert s.step(max_steps=k)[0] == k
            out.append((s.download(), s.time()))
    for Q, t in out[1:]:
        assert np.array_equal(Q, out[0][0]) and t == out[0][1]


def test_two_phase_stop_and_profile(hyp):
    from hyperelasticsolver_gb300 import HyperelasticityMPh as HM
    eos = (hyp.Barton2009(), hyp.Barton2009(_b0=2.1 * 0.1 ** 0.5))
    Ql, Qr = HM.initial_states(eos, 6)
    ref = []
    with hyp.Solver(eos, 100, model="multi", flux="hll") as s:
        s.init_riemann(Ql, Qr)
        for _ in range(20):
            ref.append((s.step(max_steps=1)[1], s.download()))
    for stop in (1, 2, 3, 13):
        with hyp.Solver(eos, 100, model="multi", flux="hll") as s:
            s.init_riemann(Ql, Qr)
            t_end = 0.5 * (ref[stop - 2][0] + ref[stop - 1][0]) if stop > 1 else 0.5 * ref[0][0]
            assert s.step(t_end=t_end) == (stop, ref[stop - 1][0])
            assert s.step(max_steps=20, t_end=t_end)[0] == 0
            s.set_profiling(True)
            s.step(max_steps=2)
            s.set_profiling(False)
            assert s.step(max_steps=18 - stop)[1] == ref[19][0]
            assert np.array_equal(s.download(), ref[19][1])
