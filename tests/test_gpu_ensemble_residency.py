"""qgn_ens_set_tiles' CTAs per SM on the x pass: no more than that many are resident on an SM, and as
many as that where the pass's own registers, threads and shared memory allow them.
"""
import ctypes as C

import pytest

from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.inputs import exponential_stratification
from qgn_fortran_b200.model import QGNEnsemble

pytestmark = pytest.mark.gpu


def residency(ens):
    n = C.c_int()
    assert ens.lib.qgn_ens_debug_residency(ens.ens, C.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("precision,threads,elements", [("fp64", 96, 16), ("fp64", 384, 8), ("mixed", 96, 32),
                                                        ("mixed", 192, 16)])
def test_x_pass_limit_is_the_resident_ctas(cuda_ok, precision, threads, elements):
    H, S, U = exponential_stratification(2)
    p = dict(nx=128, ny=128, nz=2, Lx=2.0e6, Ly=2.0e6, Htot=4000.0, C_d=0.0, TOL=1.0e30, is_explicit=True)
    ens = QGNEnsemble([QGNModule(p, H, S, U, scheme="bsrk3")], precision=precision)
    ens.set_tiles("xpass", threads, elements, 0)
    free = residency(ens)
    for k in (1, 2, 3, 4, 5, 8, 16):
        ens.set_tiles("xpass", threads, elements, k)
        assert residency(ens) == min(k, free), k
    ens.close()
