"""Device contexts set up while the process is busy elsewhere on the GPU (nothing of a
context may depend on the legacy default stream, which its own stream does not wait for),
and in one CUDA context after another."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def one_step(lib, case, dirname, storage):
    s = Solver.from_case(case, dirname, lib=lib, coherence=abi.NO_COHERENCE, storage=storage)
    try:
        dt = s.run(1)
        s.pull()
        return [dt] + [s.field(n).copy() for n in ("ux", "uy", "uz", "p", "psi", "t")]
    finally:
        s.release()


# radial lines that fill their lanes and lines that do not (whose factor rows are
# padded), per-column solves, lengths with and without powers of two
@pytest.mark.parametrize("nx,ny,nz,storage", [(64, 16, 16, 8), (70, 12, 20, 8), (300, 8, 8, 8), (600, 8, 8, 8),
                                              (64, 16, 16, 4), (40, 12, 8, 4)])
def test_set_up_beside_a_busy_default_stream(lib, tmp_path, nx, ny, nz, storage):
    import torch
    case = ic.taylor_couette(nx, ny, nz, 3400.0)
    want = one_step(lib, case, str(tmp_path / "quiet"), storage)
    stop = threading.Event()

    def keep_busy():   # two short kernels queued at any time, at most 400
        queued = []
        for _ in range(400):
            if stop.is_set():
                break
            torch.cuda._sleep(10_000_000)
            queued.append(torch.cuda.Event())
            queued[-1].record()
            if len(queued) > 2:
                queued.pop(0).synchronize()

    busy = threading.Thread(target=keep_busy)
    busy.start()
    try:
        got = one_step(lib, case, str(tmp_path / "busy"), storage)
    finally:
        stop.set()
        busy.join()
        torch.cuda.synchronize()
    for w, g in zip(want, got):
        assert np.isfinite(g).all() and np.array_equal(w, g)   # the same kernels on the same values


CHILD = """
import ctypes as C, dataclasses, sys, tempfile
import numpy as np
sys.path.insert(0, sys.argv[1])
from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

cu, lib = C.CDLL("libcuda.so.1"), abi.load()

def ok(status):
    assert status == 0, status

def steps():
    out = []
    for make, n, implicit, storage in ((ic.taylor_couette, (64, 16, 16), "x", 8), (ic.taylor_couette, (256, 12, 20), "x", 8),
                                       (ic.plane_couette, (320, 32, 16), "xyz", 8), (ic.taylor_couette, (96, 16, 16), "x", 4)):
        case = dataclasses.replace(make(*n, 500.0), implicit=tuple(d in implicit for d in "xyz"))
        with tempfile.TemporaryDirectory() as d:
            s = Solver.from_case(case, d, lib=lib, coherence=abi.NO_COHERENCE, storage=storage)
        out.append(s.run(3))
        s.pull()
        out += [s.field(f).copy() for f in ("ux", "uy", "uz", "p", "t")]
        s.release()
    return out

ok(cu.cuInit(0))
dev, runs = C.c_int(), []
ok(cu.cuDeviceGet(C.byref(dev), 0))
for _ in range(2):
    ctx = C.c_void_p()
    ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, dev))
    runs.append(steps())
    ok(cu.cuCtxDestroy_v2(ctx))
runs.append(steps())     # the device's primary context
for r in runs[1:]:
    for a, b in zip(runs[0], r):
        assert np.isfinite(b).all() and np.array_equal(a, b)
print("same in every context")
"""


def test_one_cuda_context_after_another():
    """The kernels' shared-memory limits belong to a CUDA context: a process that makes
    another one current on the same device (or resets it) gets them set again."""
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same in every context" in r.stdout, r.stdout + r.stderr
