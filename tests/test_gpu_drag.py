"""Quadratic drag: its transforms are extra tiles of the x pass (the bottom layer's u and v once
more) and a second pair of y transforms in the bottom layer's tiles.  Grids with fewer row pairs
than a CTA takes (16 and 32 points), every x-pass width (one thread to one warp per transform, 2048
points across warps) and two layers, where half the tiles are the bottom layer's.  Tolerances as for
the other right-hand-side tests: 1e-12 per layer in FP64, 1e-5 for FP32 transforms (2048 points).
"""
import numpy as np
import pytest

from oracle.qgn_oracle import Params, QGNOracle
from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 2), (32, 16, 3), (64, 256, 5), (256, 64, 2), (512, 16, 2),
                                      (1024, 64, 3), (2048, 32, 2)])
def test_drag_rhs(cuda_ok, nx, ny, nz, precision, tol):
    H, S, U = exponential_stratification(nz)
    # drag that is no small correction: its share of the bottom layer's tendency is of order one
    p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=0.0,
             A8=0.0, r0=1.0e-7, C_d=0.1, TOL=1.0e-10, is_explicit=False, dt_max=1000.0)
    m = QGNOracle(Params(**p), H, S, U)
    g = QGNModule(p, H, S, U, precision=precision)
    q = m.initialize_spec(seeded_random_pv(nx, ny, nz, 4.0, 1.0e-6, seed=nx + ny + nz))
    a, b = g.get_rhs(q), m.get_rhs(q)
    err = np.linalg.norm((a - b).reshape(nz, -1), axis=1) / np.linalg.norm(b.reshape(nz, -1), axis=1)
    assert np.all(err <= tol), err
