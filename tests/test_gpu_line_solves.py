"""The implicit line solves at the edges of their kernels: periodic y and z lines on
both sides of every number of elements per lane (and beyond the longest), radial lines
longer than a CTA likewise, tiles of radial indices that are partly empty, and the
implicit masks that end in each direction (whose solve stores the updated fields),
against the numpy oracle."""
import dataclasses

import numpy as np
import pytest

from oracle import tc_numpy as tn
from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

pytestmark = pytest.mark.gpu

T, F = True, False
SHAPES = [
    (17, 4, 32, (T, T, T)), (16, 32, 36, (F, T, T)), (18, 34, 64, (T, F, T)), (2, 66, 96, (F, F, T)),
    (33, 64, 4, (T, T, F)), (5, 98, 128, (T, T, T)), (4, 130, 192, (T, T, T)), (3, 194, 256, (F, T, T)),
    (4, 256, 260, (T, T, T)), (3, 258, 384, (T, T, T)), (2, 386, 512, (T, T, T)), (4, 512, 8, (T, T, F)),
    (3, 514, 12, (T, T, T)), (4, 6, 516, (T, T, T)), (3, 1024, 8, (F, T, F)), (2, 4, 1020, (T, T, T)), (2, 1026, 8, (T, T, T)),
    (384, 6, 4, (T, F, F)), (385, 4, 4, (T, F, F)), (400, 6, 4, (T, T, T)), (512, 6, 4, (T, F, F)),
    (513, 4, 4, (T, F, F)), (768, 6, 4, (T, F, F)), (769, 4, 4, (T, F, T)), (1024, 4, 4, (T, F, F)),
]


@pytest.mark.parametrize("curved", [True, False])
@pytest.mark.parametrize("nx,ny,nz,implicit", SHAPES)
def test_line_solves_match_oracle(lib, tmp_path, nx, ny, nz, implicit, curved):
    make = ic.taylor_couette if curved else ic.plane_couette
    case = dataclasses.replace(make(nx, ny, nz, 500.0), implicit=implicit)
    d0 = ic.write_ic(case, str(tmp_path / "ic"))
    prm = tn.Params(case.uy_xm, case.uy_xp, case.t_xm, case.t_xp, case.implicit, case.coef_dt_adv, case.coef_dt_dif)
    d = tn.load_domain(d0)
    fl = tn.load_fluid(d, d0, case.Re, case.Pr, prm)
    dt = tn.decide_dt(d, fl, prm)
    for rk in range(2):
        tn.predict_field(d, rk, dt, fl, prm)
    # the stage parity tests' tolerances: FP64, and fields rounded to 32 bits
    for storage, tol in ((8, 1e-12), (4, 1e-5)):
        s = Solver.from_ic(d0, case=case, lib=lib, coherence=abi.NO_COHERENCE, storage=storage)
        try:
            s.push()
            for rk in range(2):
                s.predict(rk, dt)
            s.pull()
            for n in ("ux", "uy", "uz", "t"):
                want = getattr(fl, n)[:, :, 1:] if n == "ux" else getattr(fl, n)
                got = s.field(n)
                assert np.all(np.isfinite(got)), (n, storage)
                assert np.abs(got - want).max() <= tol * max(np.abs(want).max(), 1e-300), (n, storage)
        finally:
            s.release()
