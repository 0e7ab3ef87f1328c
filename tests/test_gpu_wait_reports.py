"""A bounded wait that runs out in one launch of an update is reported by that
update, whichever launch it is: the right-hand side (whose record the plain
solve's semi-iteration reads with its first residual), or a step of a solve
that ends on its bound, with no residual pass after it.  The launch's loader
stops before its fourth load, the waits are bounded at about a millisecond,
nothing faults, and the context then runs a clean step.  In the precision form
a Chebyshev step of an update that ends on its prediction.

The same of a Gauss projection, whose second launch here repeats the first one
up to the sweep that met the tolerance: messages withheld in either are an
error, with the field as it was."""
import ctypes

import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, _capi, lattice, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
M, C = 1.0, [1.0, 1.0, 1.0, 1.0]


def update(h, g):
    st = _capi.CnStats()
    c = _capi.coeffs(C)
    rc = _capi.load().nrq_heavy_update_cn(nrqcd.solver_handle(), h.handle, g.handle, M, _capi.dptr(c), 1.0,
                                          ctypes.byref(st))
    return rc, st.as_dict()


def check_one_launch(oracle, form, tol, launch, before):
    """`before` clean updates, one with launch number `launch` stalled, then clean fields on the same solver."""
    n = (8, 6, 4)
    links, ef = oracle.transverse_box(n, A, 3.0, 1.0, 0.0, 5, identity_links=False)
    with lattice_ctx(n, A, cn=(M, C, 1.0, tol, 10000, form)):
        nrqcd.SetStencil(nrqcd.STENCIL_FMA)
        if form == nrqcd.FORM_PRECISION:
            nrqcd.SetChebStencil(nrqcd.CHEB_BLOCKS)
        g = GaugeConfiguration()
        g.upload(links, ef)
        h = NRQCDField()
        h.InitSinglePoint(1, 1)
        for _ in range(before):
            rc, st = update(h, g)
            assert rc == _capi.NRQ_OK and st["converged"] == 1
        nrqcd.SetWaitTest(wait_cycles=2_000_000, stall_load=3, launch=launch)
        rc, st = update(h, g)
        nrqcd.SetWaitTest()
        assert rc == _capi.NRQ_ERR_TIMEOUT and st["converged"] == 0, (rc, st)
        assert b"wait" in _capi.load().nrq_last_error(lattice.context())
        q, an = oracle.single_point(n, 1), oracle.single_point(n, 1)
        h.upload(q, an)
        rc, st = update(h, g)
        assert rc == _capi.NRQ_OK and st["converged"] == 1
        gq, ga = h.download()
        oracle.cn_update(n, A, links, ef, M, C, 1.0, q, an, tol=1e-14)
        assert np.abs(gq - q).max() < 50 * tol and np.abs(ga - an).max() < 50 * tol


@pytest.mark.parametrize("before", [0, 1, 3])
def test_right_hand_side(oracle, before):
    check_one_launch(oracle, nrqcd.FORM_PLAIN_FP64, 1e-12, 0, before)


# launch 0 the right-hand side, 1 the first residual, then the steps
@pytest.mark.parametrize("launch", [2, 4])
def test_step_of_an_unconfirmed_solve(oracle, launch):
    check_one_launch(oracle, nrqcd.FORM_PLAIN_FP64, 1e-12, launch, 2)


# launch 0 the right-hand side, 1 the residual, then the steps
@pytest.mark.parametrize("launch", [2, 4])
def test_step_of_a_predicted_update(oracle, launch):
    check_one_launch(oracle, nrqcd.FORM_PRECISION, 1e-10, launch, 6)


@pytest.mark.parametrize("launch", [0, 1])
def test_gauss_projection(oracle, launch):
    n, a = (5, 4, 3), (0.1, 1.0, 1.0, 1.0)
    links, ef = oracle.transverse_box(n, a, 2.0, 1.0, 0.0, 9, identity_links=False)
    ef = ef + 0.02 * np.random.default_rng(4).standard_normal(ef.shape)
    with lattice_ctx(n, a, cn=(M, C, 1.0, 1e-12)):
        g = GaugeConfiguration()

        def project(tol, limit):
            sweeps, dev = ctypes.c_int64(), ctypes.c_double()
            g.upload(links, ef)
            rc = _capi.load().nrq_gauge_gauss_project(g.handle, tol, limit, ctypes.byref(sweeps), ctypes.byref(dev))
            return rc, sweeps.value, dev.value

        rc, sweeps, dev = project(1e-9, 5)
        assert rc == _capi.NRQ_ERR_NOT_CONVERGED and sweeps == 5
        tol = dev * (1 + 1e-9)  # met after the fifth sweep
        nrqcd.SetWaitTest(wait_cycles=2_000_000, projection=launch)
        rc, _, _ = project(tol, 0)
        nrqcd.SetWaitTest()
        assert rc == _capi.NRQ_ERR_TIMEOUT
        assert np.array_equal(g.download()[1], ef)
        assert project(tol, 0)[:2] == (_capi.NRQ_OK, 5)
        got = g.download()[1]
    want, l = ef.copy(), links.copy()
    oracle.gauss_project(n, a, l, want, tol=1e-9, max_sweeps=5)
    assert np.abs(got - want).max() < 1e-13 * np.abs(want).max()
