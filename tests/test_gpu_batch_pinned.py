"""Mixed batches into and out of page-locked arrays (the upload's kernel reads the array in
place, a download of 64 MB or more goes row by row) against pageable ones: the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[3], [3, 253, 254, 255, 508, 509, 1017], [300001, 17, 299000]])  # the last: 67 MB
def test_page_locked_arrays_give_the_same_bits(hyp, sizes):
    torch = pytest.importorskip("torch")
    from hyperelasticsolver_gb300._cases import batch_fill, batch_prims
    eos, n = hyp.Barton2009(), sum(sizes)
    l, r = batch_prims(eos, len(sizes), seed=4)
    Q = batch_fill(hyp.Hyperelasticity.prim2cons(eos, l), hyp.Hyperelasticity.prim2cons(eos, r), np.array(sizes))
    locked = torch.empty((14, n), dtype=torch.float64, pin_memory=True)
    locked.copy_(torch.from_numpy(Q))
    out = torch.zeros((14, n), dtype=torch.float64, pin_memory=True)
    with hyp.Batch(eos, sizes, precision="mixed") as b:
        b.upload(Q)
        b.step(2)
        a = b.download()
        b.upload(locked.numpy())
        b.step(2)
        assert np.array_equal(b.download(out.numpy()), a)
        assert np.array_equal(b.download(), a)
