"""Uploads to mixed-precision contexts and batches from an array that is page-locked in part
only: not read in place by a kernel, which would read past the mapping (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["solver", "batch"])
@pytest.mark.parametrize("part", [1, 2, 3])  # of four quarters, the first ones
def test_part_registered_array(hyp, kind, part):
    """The copy of such an array is refused by the runtime, and the context goes on; the same
    array registered as a whole, or not at all, gives the same bits."""
    torch = pytest.importorskip("torch")
    from hyperelasticsolver_gb300._cases import segment_fill, segment_states
    eos, n = hyp.Barton2009(), 1 << 14
    Q = segment_fill(hyp.Hyperelasticity.prim2cons(eos, segment_states(eos, 8)), n)
    page = 4096
    raw = np.empty(Q.nbytes + page, np.uint8)
    at = -raw.ctypes.data % page
    arr = raw[at:at + Q.nbytes].view(np.float64).reshape(Q.shape)
    arr[...] = Q
    rt = torch.cuda.cudart()
    assert Q.nbytes % (4 * page) == 0

    def stepped(c):
        c.upload(arr)
        c.step(3)
        return c.download()

    make = (lambda: hyp.Solver(eos, n, precision="mixed")) if kind == "solver" else (lambda: hyp.Batch(eos, [n], precision="mixed"))
    with make() as c:
        ref = stepped(c)
        assert int(rt.cudaHostRegister(arr.ctypes.data, part * Q.nbytes // 4, 0)) == 0
        try:
            with pytest.raises(hyp._lib.HypError):
                c.upload(arr)
        finally:
            assert int(rt.cudaHostUnregister(arr.ctypes.data)) == 0
        assert np.array_equal(stepped(c), ref)
        assert int(rt.cudaHostRegister(arr.ctypes.data, Q.nbytes, 0)) == 0
        try:
            assert np.array_equal(stepped(c), ref)
        finally:
            assert int(rt.cudaHostUnregister(arr.ctypes.data)) == 0
