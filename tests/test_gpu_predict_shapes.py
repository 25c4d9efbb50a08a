"""The predict kernel at the edges of its instances: radial lengths around each
warp count (odd ones included, and tiles of longer lines), line counts that leave
the last block partly empty, single planes, and every implicit mask, against the
numpy oracle (three substeps of the predict alone, so that the previous source
terms take part)."""
import dataclasses

import numpy as np
import pytest

from oracle import tc_numpy as tn
from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

pytestmark = pytest.mark.gpu

X, XYZ, NONE, Y = (True, False, False), (True, True, True), (False,) * 3, (False, True, False)
SHAPES = [
    (2, 4, 4, X), (3, 6, 4, NONE), (31, 10, 4, X), (32, 8, 8, X), (33, 6, 12, X), (64, 10, 4, XYZ), (65, 4, 8, X),
    (95, 6, 4, X), (97, 10, 4, X), (128, 14, 4, NONE), (129, 4, 8, X), (192, 6, 8, XYZ), (193, 4, 4, X),
    (255, 6, 8, X), (256, 4, 16, Y), (257, 4, 4, X), (319, 6, 8, X), (512, 4, 4, NONE),
]


def run_oracle(case, d0):
    prm = tn.Params(case.uy_xm, case.uy_xp, case.t_xm, case.t_xp, case.implicit, case.coef_dt_adv, case.coef_dt_dif)
    d = tn.load_domain(d0)
    fl = tn.load_fluid(d, d0, case.Re, case.Pr, prm)
    dt = tn.decide_dt(d, fl, prm)
    for rk in range(3):
        tn.predict_field(d, rk, dt, fl, prm)
    return dt, fl


@pytest.mark.parametrize("curved", [True, False])
@pytest.mark.parametrize("nx,ny,nz,implicit", SHAPES)
def test_predict_edges_match_oracle(lib, tmp_path, nx, ny, nz, implicit, curved):
    make = ic.taylor_couette if curved else ic.plane_couette
    case = dataclasses.replace(make(nx, ny, nz, 500.0), implicit=implicit)
    d0 = ic.write_ic(case, str(tmp_path / "ic"))
    dt, fl = run_oracle(case, d0)
    # the FP64 tolerance is that of the stage parity tests; single storage rounds
    # the fields and source terms three times (2^-24 each) and sums about 50 rounded terms
    for storage, tol in ((8, 1e-12), (4, 1e-5)):
        s = Solver.from_ic(d0, case=case, lib=lib, coherence=abi.NO_COHERENCE, storage=storage)
        try:
            s.push()
            for rk in range(3):
                s.predict(rk, dt)
            s.pull()
            for n in ("ux", "uy", "uz", "t"):
                want = getattr(fl, n)[:, :, 1:] if n == "ux" else getattr(fl, n)
                got = s.field(n)
                assert np.all(np.isfinite(got)), (n, storage)
                assert np.abs(got - want).max() <= tol * max(np.abs(want).max(), 1e-300), (n, storage)
        finally:
            s.release()
