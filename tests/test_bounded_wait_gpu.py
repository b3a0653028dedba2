"""The device-side bounded wait, the grid barrier of the small-lattice CG: with
an arrival missing every block leaves after the time limit, the host gets
IRO_TIMEOUT, and the context keeps working."""
import ctypes

import numpy as np
import pytest

import iroiro_b200 as ib
from conftest import TOL_FP64, TOL_RES, TOL_SOL, load_golden, rel

pytestmark = pytest.mark.gpu


def test_wait_runs_out_and_context_stays_usable(port):
    g = load_golden("4x4x4x4")
    c = ib.context(g["L"])
    c.upload_gauge(g["u"], force=True)
    waited = ctypes.c_double(0.0)
    for limit in (20.0, 50.0):
        rc = c._lib.iro_selftest_bounded_wait(c.h, limit, ctypes.byref(waited))
        assert rc == ib.TIMEOUT
        assert limit <= waited.value < limit + 200.0
    # the context and the device still work: a solve over the same barrier, and
    # an operator against the oracle
    D = ib.Dirac_Wilson_EvenOdd(float(g["mass"]), g["u"], ctx=c)
    x = np.empty_like(g["f_half"])
    assert ib.Solver_CG(1e-20, 5000, ib.Fopr_DdagD(D)).solve(x, g["f_half"]).diff < TOL_RES
    assert rel(x, g["cg_wilson_eo_x"]) < TOL_SOL
    m = float(g["mass"])
    f = g["f_half"]
    assert rel(c.apply(ib.OP_WILSON_SCHUR_EE, m, 0.0, 0, f),
               port.wilson_eo(g["L"], g["u"], m, 0, f)) < TOL_FP64


@pytest.mark.parametrize("inner", ["double", "single", "half"])
def test_solve_whose_barrier_runs_out_is_done_launched(inner):
    """A small-lattice CG that gives up at its barrier is the launched solve, bit
    for bit, and the next solve is the one-launch one again."""
    g = load_golden("4x4x4x4")
    c = ib.context(g["L"])
    D = ib.Dirac_Wilson_EvenOdd(float(g["mass"]), g["u"], ctx=c)
    b = g["f_half"]
    solve = lambda **kw: ib.Solver_CG(1e-20, 5000, ib.Fopr_DdagD(D), inner=inner, **kw).solve_many(b, 1)
    launched, small = solve(launched=True)[0], solve()[0]
    assert c._lib.iro_selftest_cg_timeout(c.h, 20.0) == ib.OK
    x, outs, rc = solve()
    assert rc == ib.OK and outs[0].diff < TOL_RES and outs[0].timing >= 20.0
    assert np.array_equal(x, launched)
    x, outs, rc = solve()
    assert rc == ib.OK and np.array_equal(x, small) and outs[0].timing < 20.0


def test_wait_limit_is_checked():
    g = load_golden("4x4x4x4")
    c = ib.context(g["L"])
    waited = ctypes.c_double(0.0)
    for bad in (0.0, -1.0, 1001.0):
        assert c._lib.iro_selftest_bounded_wait(c.h, bad, ctypes.byref(waited)) == ib.BAD_ARG
        assert c._lib.iro_selftest_cg_timeout(c.h, bad) == ib.BAD_ARG
