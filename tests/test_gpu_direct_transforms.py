"""The direct transforms of FP32-storage contexts with every number of lines per CTA
(1, 2, 4, 8, last groups partly empty, the longest lines), against the numpy oracle."""
import numpy as np
import pytest

from oracle import tc_numpy as tn
from simpletcsolver_b200 import abi, ic
from simpletcsolver_b200.solver import Solver

pytestmark = pytest.mark.gpu

SHAPES = [(5, 6, 12), (60, 30, 20), (61, 30, 20), (40, 1000, 12), (16, 100, 500), (3, 12, 2044), (5, 2046, 60)]


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
    s = Solver.from_ic(d0, case=case, lib=lib, coherence=abi.NO_COHERENCE, storage=4)
    try:
        s.push()
        s.compute_potential(0, dt)
        s.pull(abi.PSI)
        got = s.field("psi")
        inner = got[1:-1, 1:-1, 1:-1]
        # 2^-24 per stored spectral value, amplified by at most the transforms' growth;
        # the singular mode's constant is free
        assert np.abs((inner - inner.mean()) - (want - want.mean())).max() <= 2e-4 * np.abs(want - want.mean()).max()
        np.testing.assert_array_equal(got[1:-1, 1:-1, 0], got[1:-1, 1:-1, 1])
        np.testing.assert_array_equal(got[1:-1, 1:-1, -1], got[1:-1, 1:-1, -2])
        np.testing.assert_array_equal(got[:, 0], got[:, -2])
        np.testing.assert_array_equal(got[0], got[-2])
        np.testing.assert_array_equal(got[-1], got[1])
    finally:
        s.release()
