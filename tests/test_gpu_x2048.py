"""The x pass of 2048-point rows in its two forms: CTA counts (row pairs times layers, plus one layer with
quadratic drag) on both sides of the lines between them, in FP64 and with FP32 transforms, against the
oracle at the suite's bounds for right-hand sides (1e-12, and 1e-5 with FP32 transforms).
"""
import numpy as np
import pytest

from oracle.qgn_oracle import Params, QGNOracle
from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz,C_d", [(16, 2, 0.0), (64, 4, 0.0), (64, 4, 0.05), (64, 5, 0.0), (64, 9, 0.0), (64, 10, 0.0),
                                       (64, 14, 0.0), (64, 18, 0.0), (64, 18, 0.05), (64, 19, 0.0)])
def test_both_forms(cuda_ok, ny, nz, C_d):
    nx = 2048
    H, S, U = exponential_stratification(nz)
    p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=0.0,
             A8=1.0e20, r0=1.0e-7, C_d=C_d, TOL=1.0e-10, is_explicit=False, dt_max=1000.0)
    m = QGNOracle(Params(**p), H, S, U)
    q = m.initialize_spec(seeded_random_pv(nx, ny, nz, 4.0, 1.0e-6, seed=ny + nz))
    want = m.get_rhs(q)
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        g = QGNModule(p, H, S, U, precision=precision)
        got = g.get_rhs(q)
        g.cleanup()
        err = np.linalg.norm((got - want).reshape(nz, -1), axis=1) / np.linalg.norm(want.reshape(nz, -1), axis=1)
        assert np.all(err <= tol), (precision, err)
