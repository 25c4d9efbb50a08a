"""The Poisson solver at lengths that take its mixed-radix transforms (every radix,
primes summed directly, one-line blocks) and at radial lengths around the lanes'
element counts of the warp solves (and past them), against the numpy oracle."""
import numpy as np
import pytest

from oracle import tc_numpy as tn
from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

pytestmark = pytest.mark.gpu

SHAPES = [
    (5, 12, 20), (7, 10, 28), (12, 14, 44), (16, 22, 52), (9, 26, 36), (6, 34, 60), (4, 46, 76), (8, 18, 100),
    (3, 1022, 4), (2, 4, 508), (4, 2046, 4), (8, 180, 120), (33, 6, 12), (64, 12, 8), (96, 8, 12), (100, 10, 4),
    (129, 4, 12), (192, 6, 4), (200, 4, 4), (257, 6, 4), (384, 4, 4), (385, 4, 8), (512, 6, 4), (520, 4, 4),
]


@pytest.mark.parametrize("nx,ny,nz", SHAPES)
def test_potential_matches_oracle(lib, tmp_path, nx, ny, nz):
    case = ic.taylor_couette(nx, ny, nz, 500.0)
    d0 = ic.write_ic(case, str(tmp_path / "ic"))
    d = tn.load_domain(d0)
    prm = tn.Params(case.uy_xm, case.uy_xp, case.t_xm, case.t_xp, case.implicit, case.coef_dt_adv, case.coef_dt_dif)
    fl = tn.load_fluid(d, d0, case.Re, case.Pr, prm)
    dt = tn.decide_dt(d, fl, prm)
    tn.compute_potential(d, 0, dt, fl)
    want = fl.psi[1:-1, 1:-1, 1:-1]
    # FP64: the bound of the stage parity tests for psi; single storage: 2^-24 per
    # stored spectral value, amplified by at most the transforms' growth
    for storage, tol in ((8, 1e-11), (4, 2e-4)):
        s = Solver.from_ic(d0, case=case, lib=lib, coherence=abi.NO_COHERENCE, storage=storage)
        try:
            s.push()
            s.compute_potential(0, dt)
            s.pull(abi.PSI)
            got = s.field("psi")
            inner = got[1:-1, 1:-1, 1:-1]
            # the singular mode's constant is free
            assert np.abs((inner - inner.mean()) - (want - want.mean())).max() <= tol * np.abs(want - want.mean()).max()
            np.testing.assert_array_equal(got[1:-1, 1:-1, 0], got[1:-1, 1:-1, 1])
            np.testing.assert_array_equal(got[1:-1, 1:-1, -1], got[1:-1, 1:-1, -2])
            np.testing.assert_array_equal(got[:, 0], got[:, -2])
            np.testing.assert_array_equal(got[0], got[-2])
            np.testing.assert_array_equal(got[-1], got[1])
        finally:
            s.release()
