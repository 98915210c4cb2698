"""GetPsi over the layer counts where its kernel changes: one thread per mode up to 8 layers, the
FP64 matrix-unit contractions (layers padded to 16, 24 or 32) above.  The grids' mode counts
(10 x 21, 21 x 10, 10 x 170) are no multiples of the four modes of a matrix row block or of the 64
of a CTA.  Tolerances: a sum of nz <= 32 products in any order is within nz eps = 7e-15 of the
exact one relative to the sum of its terms' sizes; the modal amplitudes of these fields lose at most
two digits to cancellation, so 1e-12 per layer, as for the other FP64 tests.  The mixed mode stores
q and psi in FP32: 2e-6 for one right-hand side, as in tests/test_gpu_mixed.py.
"""
import numpy as np
import pytest

from oracle.qgn_oracle import Params, QGNOracle, SCHEMES
from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu


def layer_rel(a, b):
    return np.linalg.norm((a - b).reshape(len(a), -1), axis=1) / np.linalg.norm(b.reshape(len(b), -1), axis=1)


def model(nx, ny, nz, scheme="ark43_qgleith", precision="fp64", **kw):
    H, S, U = exponential_stratification(nz, ratio=1.1)
    p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=0.0,
             A8=1.0e20, r0=1.0e-7, C_d=0.0, TOL=1.0e30, is_explicit=False, dt_max=2000.0)
    p.update(kw)
    m = QGNOracle(Params(**p), H, S, U)
    q = m.initialize_spec(seeded_random_pv(nx, ny, nz, 4.0, 1.0e-6, seed=nx + ny + nz))
    return m, QGNModule(p, H, S, U, scheme=scheme, precision=precision), q


@pytest.mark.parametrize("nz", [2, 3, 5, 6, 7, 8, 9, 12, 15, 16, 17, 23, 24, 25, 31, 32])
@pytest.mark.parametrize("nx,ny", [(32, 32), (64, 16), (32, 256)])
def test_get_psi(cuda_ok, nx, ny, nz):
    m, g, q = model(nx, ny, nz)
    assert np.all(layer_rel(g.get_psi(q), m.get_psi(q)) <= 1e-12)
    assert g.get_psi(q)[:, 0, 0].tolist() == [0.0] * nz


@pytest.mark.parametrize("nz", [3, 6, 9, 16, 20, 32])
def test_mixed_rhs(cuda_ok, nz):
    m, g, q = model(64, 64, nz, precision="mixed")
    assert np.all(layer_rel(g.get_rhs(q), m.get_rhs(q)) <= 2e-6)


@pytest.mark.parametrize("nz", [3, 8, 9, 32])
@pytest.mark.parametrize("scheme", ["bsrk3", "rk4", "ab3", "ark43"])
def test_steps(cuda_ok, scheme, nz):
    """The explicit schemes' combinations (with GetPsi up to 8 layers) and ARK43's stages."""
    m, g, q = model(64, 32, nz, scheme=scheme, is_explicit=scheme != "ark43")
    st = SCHEMES[scheme](m)
    qg, t, dt = q.copy(), 0.0, 2000.0
    want, tw, dw = q, 0.0, 2000.0
    for _ in range(3):
        t, dt = g.time_step(qg, t, dt)
        want, tw, dw = st.step(want, tw, dw)
    assert (t, dt) == (tw, dw)
    assert np.all(layer_rel(qg, want) <= 1e-12)
