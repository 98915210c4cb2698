"""What a call reports when a bounded device wait of it ran out.

The kernels set a flag and finish; here the flag is set by hand (qgn_debug_set_wait), no wait is made
to run out.  The adaptive schemes' controller halts the run on its own flag.  Everything that has no
controller -- right-hand sides, physical fields, training samples, the fixed-step schemes -- reports
the context's other flag as QGN_ERR_CUDA, once, and leaves the run alone.
"""
import ctypes as C

import numpy as np
import pytest

from qgn_fortran_b200 import QGNModule, _lib
from qgn_fortran_b200.inputs import exponential_stratification, seeded_random_pv

pytestmark = pytest.mark.gpu

STEP, CALL = 0, 1


def model(scheme, precision="fp64", n=64, nz=3):
    H, S, U = exponential_stratification(nz)
    p = dict(nx=n, ny=n, nz=nz, Lx=2.0e6, Ly=2.0e6, Htot=4000.0, beta=2.0e-11, A8=1.0e20, r0=1.0e-7, C_d=0.0,
             TOL=1.0e30, is_explicit=scheme in ("rk4", "ab3", "bsrk3"), dt_max=900.0)
    g = QGNModule(p, H, S, U, scheme=scheme, precision=precision)
    return g, g.initialize(seeded_random_pv(n, n, nz, 6.0, 1.0e-6, seed=7), 0.0, 900.0)


def ran_out(g, which):
    assert g.lib.qgn_debug_set_wait(g.ctx, which, 1) == 0


def fails(f, code=_lib.QGN_ERR_CUDA):
    with pytest.raises(_lib.QGNError) as ei:
        f()
    assert ei.value.code == code


@pytest.mark.parametrize("scheme,precision", [("ark43_qgleith", "fp64"), ("ark43", "mixed"), ("bsrk3", "fp64"),
                                              ("rk4", "fp64")])
def test_evaluations_report_it_once(cuda_ok, scheme, precision):
    g, q = model(scheme, precision)
    calls = [lambda: g.get_rhs(q), lambda: np.stack(g.physical(q))]
    if precision == "fp64":
        calls.append(lambda: np.stack(g.physical_modal(q)))
    for f in calls:
        want = f()
        ran_out(g, CALL)
        fails(f)
        assert np.array_equal(f(), want)
    if scheme != "rk4":   # the run's flag is the run's
        ran_out(g, STEP)
        for f in calls:
            f()
    g.cleanup()


@pytest.mark.parametrize("scheme,precision", [("ark43_qgleith", "fp64"), ("ark43", "mixed"), ("bsrk3", "fp64")])
def test_adaptive_steps_halt(cuda_ok, scheme, precision):
    g, q = model(scheme, precision)
    want, _ = model(scheme, precision)
    want.advance_resident(2)
    ran_out(g, CALL)          # not looked at by the steps
    g.advance_resident(1)
    fails(lambda: g.get_rhs(q))
    ran_out(g, STEP)
    fails(lambda: g.advance_resident(1))
    fails(lambda: g.advance_resident(1), _lib.QGN_ERR_CONFIG)
    g.set_state(q, 0.0, 900.0)
    g.advance_resident(2)
    # BSRK3 starts again from a right-hand side of the new state, the others keep none
    assert np.array_equal(g.get_state(), want.get_state())
    g.cleanup()


@pytest.mark.parametrize("scheme", ["rk4", "ab3"])
def test_fixed_steps_report_it(cuda_ok, scheme):
    g, q = model(scheme)
    want, _ = model(scheme)
    want.advance_resident(3)
    g.advance_resident(2)
    ran_out(g, CALL)
    fails(lambda: g.advance_resident(1))
    fails(lambda: g.advance_resident(1), _lib.QGN_ERR_CONFIG)
    ran_out(g, CALL)
    fails(lambda: g.advance(q.copy(), 0.0, 900.0, 1))
    g.set_state(q, 0.0, 900.0)
    g.advance_resident(3)     # AB3's history starts again
    assert np.array_equal(g.get_state(), want.get_state())
    g.cleanup()


@pytest.mark.parametrize("late", ["fine", "coarse"])
def test_training_samples_report_it(cuda_ok, late):
    import torch

    fine, _ = model("ark43_qgleith", n=256, nz=2)
    coarse, _ = model("ark43_qgleith", n=128, nz=2)
    x = torch.empty((128, 128, 16), dtype=torch.bfloat16, device="cuda")
    y = torch.empty((128, 128, 16), dtype=torch.float32, device="cuda")
    one = (C.c_float * 4)(1.0, 1.0, 1.0, 1.0)

    def snapshot():
        return fine.lib.qgn_closure_snapshot(fine.ctx, coarse.ctx, one, one, C.c_void_p(x.data_ptr()),
                                             C.c_void_p(y.data_ptr()), 16, 16)
    assert snapshot() == 0
    ran_out(fine if late == "fine" else coarse, CALL)
    assert snapshot() == _lib.QGN_ERR_CUDA
    assert snapshot() == 0
    fine.cleanup()
    coarse.cleanup()
