"""Two-phase FP64 faces whose volume fractions jump (the ones listed for their path
integrals): where they lie in a block, how many of them there are, and how many nodes they
take, against the oracle (GPU)."""
import ctypes

import numpy as np
import pytest

from helpers import RTOL_FP64, assert_close_soa
from test_gpu_two_faces import setup, smooth_state
from test_paths64_host import DEFAULT, lib, path  # noqa: F401 (lib: a fixture)

pytestmark = pytest.mark.gpu

N = 12300  # above 152 blocks of 64 cells, where LxF face blocks keep marks


def prims(orc, pb, n):
    return np.array(orc.cons2prim(pb, np.ascontiguousarray(smooth_state(orc, pb, n, False).T)))


def one_step(hyp, orc, flux, P, eos, pb):
    Q0 = np.ascontiguousarray(orc.prim2cons(pb, P).T)
    Qo, _, to, _ = orc.run(pb, Q0, max_steps=1)
    with hyp.Solver(eos, P.shape[0], model="multi", flux=flux, bc="transmissive") as s:
        s.upload(Q0)
        n, t = s.step(max_steps=1)
        assert n == 1 and abs(t - to) <= RTOL_FP64 * to
        assert_close_soa(s.download(), Qo, RTOL_FP64, flux)


def fractions(P, a):
    P[:, 0], P[:, 15] = a, 1.0 - a
    return P


@pytest.mark.parametrize("flux", ["hll", "lxf"])
def test_places_in_a_block(hyp, orc, flux):
    """Jumps at the domain's first and last inner face and on a block's first, last and middle
    slots: a few marked blocks beside unmarked ones, some next to each other."""
    eos, pb = setup(hyp, orc, N, flux, bc=orc.BC_TRANSMISSIVE)
    a = np.full(N, 0.3)
    for k, f in enumerate((1, 640, 767, 768, 1983, 6431, 6433, 9983, N - 1)):  # face f: cells f - 1, f
        a[f:] = 0.3 + 0.04 * (k + 1)
    one_step(hyp, orc, flux, fractions(prims(orc, pb, N), a), eos, pb)


@pytest.mark.parametrize("flux", ["hll", "lxf"])
@pytest.mark.parametrize("per_sm", [4, 48])  # a warp a face up to 4 a multiprocessor; a thread above 48
@pytest.mark.parametrize("more", [0, 1])
def test_list_lengths(hyp, orc, flux, per_sm, more):
    torch = pytest.importorskip("torch")
    listed = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    n = max(N, listed + 100)
    eos, pb = setup(hyp, orc, n, flux, bc=orc.BC_TRANSMISSIVE)
    a = np.full(n, 0.4)
    a[:listed] = 0.4 + 0.1 * np.sin(2 * np.pi * (1 + np.arange(listed)) / 997.0)  # the last of them jumps to 0.4
    assert np.count_nonzero(a[1:] != a[:-1]) == listed
    one_step(hyp, orc, flux, fractions(prims(orc, pb, n), a), eos, pb)


@pytest.mark.parametrize("flux", ["hll", "lxf"])
def test_node_counts(hyp, orc, lib, flux):  # noqa: F811
    """A list of all faces, so a thread each, whose first integrals take 2, 3 and 6 nodes: waves
    of amplitudes from 1e-8 up, and fractions that hardly jump between states that do."""
    eos, pb = setup(hyp, orc, N, flux, bc=orc.BC_TRANSMISSIVE)
    x = (np.arange(N) + 0.5) / N
    amp = 10.0 ** (-8 + 7 * x)
    P = prims(orc, pb, N)
    mean = np.mean(P, axis=0)
    wig = np.sin(2 * np.pi * 1500 * x)[:, None] * np.linspace(-1, 1, 30)[None, :]
    P = np.where(np.arange(30) % 15 == 5, mean, mean + (0.2 * amp)[:, None] * wig)  # (entropies stay)
    a = 0.4 + 0.1 * amp * np.sin(2 * np.pi * 1500 * x + 1.0)
    tail = slice(9 * N // 10, N)
    a[tail] = 0.4 * (1 + 1e-9 * np.arange(N)[tail])
    for p in (0, 15):
        P[:, p + 1] = 8.93 / np.linalg.det(P[:, p + 6:p + 15].reshape(-1, 3, 3))
    P = fractions(P, a)
    assert np.all(a[1:] != a[:-1])
    Q = np.asarray(orc.prim2cons(pb, P))
    nodes = [path(lib, DEFAULT, Q[f - 1], Q[f])[0] for f in range(1, N, 5)]
    assert min(nodes.count(k) for k in (2, 3, 6)) > 50, [nodes.count(k) for k in (2, 3, 6)]
    one_step(hyp, orc, flux, P, eos, pb)
