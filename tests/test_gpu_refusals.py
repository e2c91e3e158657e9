"""FP64 runs where the runtime refuses something (GPU): a cooperative launch, where the process
may not have all its blocks at once (the steps then run as kernels of their own), or a second
flux buffer, where there is no room for one (the step's kernels then run apart). The refusals
are fakes: the library's own objects, linked with calls that return the error."""
import glob
import os
import subprocess
import sys

import numpy as np
import pytest

from hyperelasticsolver_gb300 import _cases as C
from hyperelasticsolver_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FAKE = """
#include <stdio.h>
#include <stdlib.h>
static int refuse(int error) {
  fputs("refused\\n", stderr);
  return error;
}
int __real_cudaMalloc(void**, size_t);
int __wrap_cudaLaunchCooperativeKernel(void) { return refuse(720); }  /* too large */
static int seen;
int __wrap_cudaMalloc(void** p, size_t n) {  /* no memory for the second buffer of that size */
  const char* e = getenv("NO_SECOND_OF");
  return e && n == (size_t)atoll(e) && ++seen == 2 ? refuse(2) : __real_cudaMalloc(p, n);
}
"""
CHILD = """
import ctypes, sys
import numpy as np, torch
import hyperelasticsolver_gb300 as hyp
hyp._lib._build.LIB = sys.argv[1]
q = np.load(sys.argv[2])
n, out = q.shape[1], {}
with hyp.Solver(hyp.Barton2009(), n) as s:
    s.upload(q)
    out["steps"] = [s.step(max_steps=20)[0], s.step(t_end=1.5 * s.time()[0])[0]]
    out["Q"], out["t"] = s.download(), s.time()[0]
for k in (7, 8):
    cfg = hyp._model.config(hyp.Barton2009(), hyp._lib.HYP_MODEL_SINGLE, n_cells=n, cfl=0.5)
    a = torch.from_numpy(q).cuda()
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    t = ctypes.c_double()
    rc = hyp._lib.load().hyp_step_noalloc_f64(cfg, a.data_ptr(), b.data_ptr(), n, k, 0.0, None, ctypes.byref(t), None)
    assert rc == 0, rc
    out[f"b{k}"], out[f"t{k}"] = b.cpu().numpy(), t.value
np.savez(sys.argv[3], **out)
"""


@pytest.fixture(scope="module")
def refusing(tmp_path_factory):
    B.build()
    d = tmp_path_factory.mktemp("refused")
    (d / "fake.c").write_text(FAKE)
    objs = sorted(glob.glob(os.path.join(B.OUT, "*.o")))
    assert objs
    lib = str(d / "lib.so")
    for cmd in (["gcc", "-fPIC", "-c", str(d / "fake.c"), "-o", str(d / "fake.o")],
                [B._nvcc(), *B.ARCH, "-shared", "-Xlinker", "--wrap=cudaLaunchCooperativeKernel",
                 "-Xlinker", "--wrap=cudaMalloc", "-o", lib, *objs, str(d / "fake.o")]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return lib


def outcomes(code, refusing, tmp_path, q, **env):
    """What the child saves with the library as it is and with the refusing one."""
    np.save(tmp_path / "q.npy", q)
    out = []
    for name, lib, e in (("own", B.LIB, {}), ("refused", refusing, env)):
        r = subprocess.run([sys.executable, "-c", code, lib, str(tmp_path / "q.npy"), str(tmp_path / name)], cwd=ROOT,
                           env={**os.environ, **e}, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0 and ("refused" in r.stderr) == (name == "refused"), r.stderr
        out.append(np.load(tmp_path / (name + ".npz")))
    for k in out[0].files:
        assert np.array_equal(out[0][k], out[1][k]), k
    return out[0]


def state(hyp, n):
    eos = hyp.Barton2009()
    return C.segment_fill(hyp.Hyperelasticity.prim2cons(eos, C.segment_states(eos, 8, seed=3)), n)


@pytest.mark.parametrize("n", [1000, 12000])
def test_refused_launch(hyp, refusing, tmp_path, n):
    pytest.importorskip("torch")
    out = outcomes(CHILD, refusing, tmp_path, state(hyp, n))
    assert out["steps"][0] == 20 and out["steps"][1] > 0


APART = """
import sys
import numpy as np
import hyperelasticsolver_gb300 as hyp
hyp._lib._build.LIB = sys.argv[1]
q = np.load(sys.argv[2])
n, out, eos = q.shape[1], {}, hyp.Barton2009()
if n % 3:
    with hyp.Solver(eos, n) as s:
        s.upload(q)
        out["steps"] = [s.step(max_steps=27)[0], s.step(t_end=1.5 * s.time()[0])[0]]
        out["Q"], out["t"] = s.download(), s.time()[0]
        s.record(9, 4)
        out["g"] = s.adjoint(q)[0]
else:
    with hyp.Batch(eos, [n // 3] * 3, precision="fp64") as b:
        b.upload(q)
        b.step(13)
        b.step(5, t_end=1.2 * b.status()[0][0])
        out["Q"], out["t"], out["steps"] = b.download(), *b.status()
np.savez(sys.argv[3], **out)
"""


@pytest.mark.parametrize("n", [30001, 30000])  # a solver, a batch of three problems
def test_no_second_flux_buffer(hyp, refusing, tmp_path, n):
    out = outcomes(APART, refusing, tmp_path, state(hyp, n), NO_SECOND_OF=str(12 * 8 * n))
    assert np.all(out["steps"] > 0)
