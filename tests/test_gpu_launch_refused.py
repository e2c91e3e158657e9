"""Small FP64 runs where the process may not have all blocks of a cooperative launch at once:
the launch is refused, and the steps run as kernels of their own (GPU). The refusal is a fake:
the library's own objects, linked with a cudaLaunchCooperativeKernel that returns the error."""
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
    (d / "fake.c").write_text("int __wrap_cudaLaunchCooperativeKernel(void) { return 720; }  /* too large */\n")
    objs = sorted(glob.glob(os.path.join(B.OUT, "*.o")))
    assert objs
    lib = str(d / "lib.so")
    for cmd in (["gcc", "-fPIC", "-c", str(d / "fake.c"), "-o", str(d / "fake.o")],
                [B._nvcc(), *B.ARCH, "-shared", "-Xlinker", "--wrap=cudaLaunchCooperativeKernel", "-o", lib, *objs, str(d / "fake.o")]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return lib


@pytest.mark.parametrize("n", [1000, 12000])
def test_steps_run_all_the_same(hyp, refusing, tmp_path, n):
    pytest.importorskip("torch")
    eos = hyp.Barton2009()
    q = C.segment_fill(hyp.Hyperelasticity.prim2cons(eos, C.segment_states(eos, 8, seed=3)), n)
    np.save(tmp_path / "q.npy", q)
    out = []
    for name, lib in (("own", B.LIB), ("refused", refusing)):
        r = subprocess.run([sys.executable, "-c", CHILD, lib, str(tmp_path / "q.npy"), str(tmp_path / name)], cwd=ROOT,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        out.append(np.load(tmp_path / (name + ".npz")))
    for k in out[0].files:
        assert np.array_equal(out[0][k], out[1][k]), k
    assert out[0]["steps"][0] == 20 and out[0]["steps"][1] > 0
