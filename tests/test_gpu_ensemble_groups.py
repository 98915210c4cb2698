"""Ensembles whose members differ in both grid lengths and in the layer count: the x pass is a launch
per grid size and every pass looks its tiles up, so members are interleaved by size here.  FP64 against
single-context BSRK3 runs (1e-12 per layer, as for the other ensemble tests), FP32 passes against the
FP64 ensemble (1e-5), with the x pass left to the tuner and limited to two CTAs per SM.
"""
import math

import numpy as np
import pytest

from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv
from qgn_fortran_b200.model import QGNEnsemble

pytestmark = pytest.mark.gpu

GRIDS = [(128, 256, 3), (256, 128, 16), (128, 128, 2), (512, 128, 7), (128, 256, 8), (256, 128, 4), (128, 128, 5)]


def members(ensemble=True):
    out = []
    for m, (nx, ny, nz) in enumerate(GRIDS):
        H, S, U = exponential_stratification(nz)
        p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=0.0,
                 A8=1.0 / (86400.0 * (math.pi * nx / 2.0e6) ** 8), r0=1.0e-7, C_d=0.0, TOL=1.0e30, is_explicit=True,
                 dt_max=900.0)
        g = QGNModule(p, H, S, U, scheme="bsrk3")
        g.initialize(seeded_random_pv(nx, ny, nz, 8.0, 1.0e-6, seed=m), 0.0, 900.0)
        out.append(g)
    return out


def rel(a, b):
    n = len(a)
    return np.max(np.linalg.norm((a - b).reshape(n, -1), axis=1) / np.linalg.norm(b.reshape(n, -1), axis=1))


@pytest.mark.parametrize("tiles", [None, (192, 16, 2)])
def test_mixed_grids(cuda_ok, tiles):
    single = members()
    for g in single:
        g.advance_resident(3)
    want = [g.get_state() for g in single]
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        ms = members()
        ens = QGNEnsemble(ms, precision=precision)
        if tiles:
            ens.set_tiles("xpass", *tiles)
        ens.advance(2)
        ens.advance(1)
        assert all(rel(g.get_state(), w) <= tol for g, w in zip(ms, want))
        assert ens.tuning()["xpass"]["threads"] in (96, 192, 384)
        ens.close()
