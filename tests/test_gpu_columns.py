"""The small grids' column path (FP64 ARK43 steps without quadratic drag: the forward x transforms stored by
column, staged by bulk copies) over the forms that its rule accepts: every built (ny, nz) edge, nx below,
at and above ny, every x-pass form, with and without the learned closure's tendency.

Against the oracle with fixed steps at the suite's bound for such trajectories (1e-11); with the closure
against the separate kernels at the suite's bound for adaptive runs (1e-9); and in the bounds-checked
build, where every global index of the column kernels is tested.
"""
import ctypes as C
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle.qgn_oracle import Params, QGNOracle, SCHEMES
from qgn_fortran_b200 import QGNModule, _lib
from qgn_fortran_b200 import closure as cl
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(16, 128, 4), (32, 128, 16), (1024, 128, 2), (2048, 128, 2), (64, 256, 4), (128, 256, 8), (512, 256, 2),
          (64, 512, 2), (64, 512, 4), (512, 512, 2)]


def parameters(nx, ny, nz, **kw):
    p = dict(nx=nx, ny=ny, nz=nz, Lx=2.0e6, Ly=2.0e6 * ny / nx, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=0.0, A8=1.0e20,
             r0=1.0e-7, C_d=0.0, TOL=1.0e30, is_explicit=False, dt_max=900.0)
    p.update(kw)
    return p


def layer_rel(a, b):
    return np.sqrt(np.sum(np.abs(a - b) ** 2, axis=(1, 2)) / np.sum(np.abs(b) ** 2, axis=(1, 2)))


def launches(g, kernel):
    k = [g.lib.qgn_kernel_name(i).decode() for i in range(_lib.QGN_KERNEL_FAMILIES)].index(kernel)
    ms, nb, timed, n = C.c_double(), C.c_double(), C.c_longlong(), C.c_longlong()
    assert g.lib.qgn_profile_read(g.ctx, k, C.byref(ms), C.byref(nb), C.byref(timed), C.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("scheme", ["ark43", "ark43_qgleith"])
@pytest.mark.parametrize("nx,ny,nz", SHAPES)
def test_against_oracle(cuda_ok, nx, ny, nz, scheme):
    H, S, U = exponential_stratification(nz)
    p = parameters(nx, ny, nz)
    m = QGNOracle(Params(**p), H, S, U)
    q = m.initialize_spec(seeded_random_pv(nx, ny, nz, 6.0, 1.0e-6, seed=nx + 7 * ny + nz))
    g = QGNModule(p, H, S, U, scheme=scheme)
    g.set_state(q, 0.0, 900.0)
    g.advance_resident(3)
    got = g.get_state()
    assert launches(g, "yinv") < launches(g, "xpass")   # the y-inverses of the stages are in the column kernels
    g.cleanup()
    st, t, dt = SCHEMES[scheme](m), 0.0, 900.0
    for _ in range(3):
        q, t, dt = st.step(q, t, dt)
    assert np.all(layer_rel(got, q) <= 1e-11)


@pytest.mark.parametrize("nx,ny,nz", [(128, 256, 2), (512, 128, 2), (128, 128, 8), (128, 512, 4)])
def test_with_closure(cuda_ok, monkeypatch, nx, ny, nz):
    H, S, U = exponential_stratification(nz)

    def run():
        g = QGNModule(parameters(nx, ny, nz, TOL=1.0e-12), H, S, U, scheme="ark43_qgleith")
        g.initialize(seeded_random_pv(nx, ny, nz, 6.0, 1.0e-6, seed=3), 0.0, 900.0)
        net = cl.ClosureNet(nz=nz, H=ny, W=nx, layers=3, max_batch=1, seed=5)
        rng = np.random.default_rng(5)
        net.set_weights([(1e-3 * rng.standard_normal(a.shape).astype(np.float32), b) for a, b in net.get_weights()])
        cl.attach(g, net, np.ones(2 * nz), np.full(nz, 1e9), A8_background=1.0e20, energy_limit=1.0)
        g.advance_resident(4)
        out = g.get_state(), g.time(), g.rejects()
        g.cleanup()
        return out
    qa, ta, ra = run()
    monkeypatch.setenv("QGN_NO_FUSED_STAGE", "1")
    qb, tb, rb = run()
    assert ra == rb and ta == pytest.approx(tb, rel=1e-9)
    assert np.all(layer_rel(qa, qb) <= 1e-9)


def checked_case(nx, ny, nz):
    """Three fixed steps: the state's norm and the failed checks (-1 in the normal build)."""
    H, S, U = exponential_stratification(nz)
    g = QGNModule(parameters(nx, ny, nz), H, S, U, scheme="ark43_qgleith")
    g.initialize(seeded_random_pv(nx, ny, nz, 6.0, 1.0e-6, seed=3), 0.0, 900.0)
    g.advance_resident(3)
    n = C.c_longlong()
    assert g.lib.qgn_check_failures(g.ctx, C.byref(n)) == 0
    out = float(np.linalg.norm(g.get_state())), n.value
    g.cleanup()
    return out


RUNNER = r'''
import json, sys
sys.path.insert(0, sys.argv[1])
from qgn_fortran_b200 import _lib
_lib.load(_lib.CHECK_LIB_PATH)
sys.path.insert(0, sys.argv[1] + "/tests")
from test_gpu_columns import SHAPES, checked_case
json.dump([checked_case(*s) for s in SHAPES], open(sys.argv[2], "w"))
'''


def test_checked_build(cuda_ok, tmp_path):
    assert os.path.exists(_lib.CHECK_LIB_PATH)
    out = tmp_path / "checked.json"
    r = subprocess.run([sys.executable, "-c", RUNNER, ROOT, str(out)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    for shape, (norm, failures) in zip(SHAPES, json.load(open(out))):
        assert failures == 0, shape
        want, _ = checked_case(*shape)          # the normal build, in this process
        assert norm == pytest.approx(want, rel=1e-11), shape
