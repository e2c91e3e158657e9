"""The bounded wait of a small FP64 run's blocks for one another (run1_f64_kernel,
run1_split_f64_kernel): it runs out without a fault, is reported, and the context goes on (GPU)."""
import numpy as np
import pytest

from hyperelasticsolver_gb300 import _cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50, 1000, 9576, 9577, 19304])  # one block; two threads a cell; one
def test_timeout_is_reported_and_recoverable(hyp, n):
    """With a poll budget of 0 every block gives up in the first step, before it has changed
    anything; with the budget restored the context steps a fresh upload as a new one does."""
    eos = hyp.Barton2009()
    Q0 = C.segment_fill(hyp.Hyperelasticity.prim2cons(eos, C.segment_states(eos, 8, seed=3)), n)
    with hyp.Solver(eos, n) as s:
        s.upload(Q0)
        s.set_wait_limit(0)
        with pytest.raises(hyp._lib.HypError) as err:
            s.step(max_steps=3)
        assert err.value.code == hyp._lib.HYP_ERR_TIMEOUT and "timed out" in str(err.value)
        assert np.array_equal(s.download(), Q0)
        s.set_wait_limit(1 << 24)
        s.upload(Q0)
        assert s.step(max_steps=20)[0] == 20
        a, ta = s.download(), s.time()
    with hyp.Solver(eos, n) as t:
        t.upload(Q0)
        t.step(max_steps=20)
        assert np.array_equal(t.download(), a) and t.time() == ta
