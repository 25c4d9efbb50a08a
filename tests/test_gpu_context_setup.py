"""Device contexts set up while the process is busy elsewhere on the GPU: nothing of a
context may depend on the legacy default stream, which its own stream does not wait for."""
import threading

import numpy as np
import pytest

from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

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
