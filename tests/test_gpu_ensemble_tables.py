"""The ensemble's tile tables go to the device when its tiles have changed, not on every advance, and a
change after steps were captured is taken up: equal to an ensemble that had the tiles from the start.
"""
import ctypes as C

import numpy as np
import pytest

from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv
from qgn_fortran_b200.model import QGNEnsemble

pytestmark = pytest.mark.gpu


def ensemble():
    ms = []
    for m, (nx, ny, nz) in enumerate([(128, 256, 3), (256, 128, 2), (128, 128, 4)]):
        H, S, U = exponential_stratification(nz)
        p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, beta=2.0e-11, A8=1.0e20, r0=1.0e-7,
                 C_d=0.0, TOL=1.0e30, is_explicit=True, dt_max=900.0)
        g = QGNModule(p, H, S, U, scheme="bsrk3")
        g.initialize(seeded_random_pv(nx, ny, nz, 6.0, 1.0e-6, seed=m), 0.0, 900.0)
        ms.append(g)
    return ms, QGNEnsemble(ms, precision="fp64")


def uploads(ens):
    n = C.c_int()
    assert ens.lib.qgn_ens_debug_uploads(ens.ens, C.byref(n)) == 0
    return n.value


def test_tables_go_up_once(cuda_ok, monkeypatch):
    monkeypatch.setenv("QGN_NO_AUTOTUNE", "1")
    tiles = (("yinv", 64, 16), ("xpass", 96, 16), ("yfwd", 64, 16))   # more tiles than the defaults
    want, ref = ensemble()
    for t in tiles:
        ref.set_tiles(*t)
    got, ens = ensemble()
    ens.advance(2)
    n = uploads(ens)
    for _ in range(3):
        ens.advance(1)
    assert uploads(ens) == n
    for m, g in enumerate(got):     # the same start again, now with other tiles
        g.set_state(want[m].get_state(), 0.0, 900.0)
    for t in tiles:
        ens.set_tiles(*t)
    for _ in range(3):
        ens.advance(1)
    assert uploads(ens) == n + 1
    ref.advance(3)
    for a, b in zip(got, want):
        assert np.array_equal(a.get_state(), b.get_state())
    ens.close()
    ref.close()
