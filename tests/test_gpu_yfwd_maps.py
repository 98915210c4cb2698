"""The y-forward pass with tensor-map rows at the sizes where its tiles change: column counts that end
inside a tile (nkx = nx/3 odd), one box and several boxes of 256 rows, FP64 and FP32 rows (two columns
are 16 bytes there), with and without the drag rows' map, and the entry point without waits, which
stages the same rows by plain loads (its y-inverse is compiled apart too, so the two agree to roundoff and
not to the bit); each against the oracle, 1e-12 per layer in FP64 and 1e-5 with FP32 transforms.
"""
import ctypes as C

import numpy as np
import pytest

from oracle.qgn_oracle import Params, QGNOracle
from qgn_fortran_b200 import QGNModule, _lib
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C_d", [0.0, 0.05])
@pytest.mark.parametrize("nx,ny,nz", [(16, 256, 3), (32, 512, 2), (64, 1024, 2), (128, 2048, 2), (512, 256, 2)])
def test_rows(cuda_ok, nx, ny, nz, C_d):
    import torch
    H, S, U = exponential_stratification(nz)
    p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=2.0,
             A8=1.0e20, r0=1.0e-7, C_d=C_d, TOL=1.0e-10, is_explicit=True, dt_max=1000.0)
    m = QGNOracle(Params(**p), H, S, U)
    q = m.initialize_spec(seeded_random_pv(nx, ny, nz, 4.0, 1.0e-6, seed=nx + ny))
    want = m.get_rhs(q)
    g = QGNModule(p, H, S, U)
    got = g.get_rhs(q)
    err = np.linalg.norm((got - want).reshape(nz, -1), axis=1) / np.linalg.norm(want.reshape(nz, -1), axis=1)
    assert np.all(err <= 1e-12), err
    p32 = dict(p, is_explicit=False)     # the mixed mode's schemes are the implicit ones
    m32, g32 = QGNOracle(Params(**p32), H, S, U), QGNModule(p32, H, S, U, precision="mixed")
    w32 = m32.get_rhs(q)
    e32 = np.linalg.norm((g32.get_rhs(q) - w32).reshape(nz, -1), axis=1) / np.linalg.norm(w32.reshape(nz, -1), axis=1)
    assert np.all(e32 <= 1e-5), e32
    # without tensor maps
    qd, out = torch.from_numpy(q).cuda(), torch.empty_like(torch.from_numpy(q)).cuda()
    torch.cuda.synchronize()
    rc = g.lib.qgn_rhs_static(C.byref(g._cp), _lib.dptr(np.ascontiguousarray(g.H)), _lib.dptr(g.uBar),
                              _lib.dptr(np.ascontiguousarray(g.qyBar)),
                              np.asfortranarray(g.Modes).ctypes.data_as(C.POINTER(C.c_double)),
                              _lib.dptr(np.ascontiguousarray(g.EVals)), C.c_void_p(qd.data_ptr()),
                              C.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    st = out.cpu().numpy()
    err = np.linalg.norm((st - want).reshape(nz, -1), axis=1) / np.linalg.norm(want.reshape(nz, -1), axis=1)
    assert np.all(err <= 1e-12), err
