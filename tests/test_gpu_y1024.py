"""The FP64 y-forward pass of 1024-point columns in its two forms (one and two columns per CTA): column counts
on both sides of the lines between them, odd ones among them, with and without quadratic drag, with tensor-map
rows and, through the entry point without waits, with plain staging loads; against the oracle at the suite's
bound for right-hand sides (1e-12).
"""
import ctypes as C

import numpy as np
import pytest

from oracle.qgn_oracle import Params, QGNOracle
from qgn_fortran_b200 import QGNModule, _lib
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,C_d", [(64, 7, 0.0), (32, 15, 0.0), (64, 8, 0.0), (64, 8, 0.05), (32, 24, 0.0), (64, 14, 0.0),
                                       (128, 7, 0.0), (256, 2, 0.0)])
def test_both_forms(cuda_ok, nx, nz, C_d):
    import torch
    ny = 1024
    H, S, U = exponential_stratification(nz)
    p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=2.0,
             A8=1.0e20, r0=1.0e-7, C_d=C_d, TOL=1.0e-10, is_explicit=True, dt_max=1000.0)
    m = QGNOracle(Params(**p), H, S, U)
    q = m.initialize_spec(seeded_random_pv(nx, ny, nz, 4.0, 1.0e-6, seed=nx + nz))
    want = m.get_rhs(q)
    g = QGNModule(p, H, S, U)
    forms = [g.get_rhs(q)]
    qd = torch.from_numpy(q).cuda()
    out = torch.empty_like(qd)
    torch.cuda.synchronize()
    rc = g.lib.qgn_rhs_static(C.byref(g._cp), _lib.dptr(np.ascontiguousarray(g.H)), _lib.dptr(g.uBar),
                              _lib.dptr(np.ascontiguousarray(g.qyBar)),
                              np.asfortranarray(g.Modes).ctypes.data_as(C.POINTER(C.c_double)),
                              _lib.dptr(np.ascontiguousarray(g.EVals)), C.c_void_p(qd.data_ptr()),
                              C.c_void_p(out.data_ptr()), None)
    if rc != _lib.QGN_ERR_TOO_LARGE:
        assert rc == 0
        torch.cuda.synchronize()
        forms.append(out.cpu().numpy())
    g.cleanup()
    for got in forms:
        err = np.linalg.norm((got - want).reshape(nz, -1), axis=1) / np.linalg.norm(want.reshape(nz, -1), axis=1)
        assert np.all(err <= 1e-12), err
