"""Each Wilson coefficient complex by itself: the spin-structured stencil and
the Chebyshev semi-iteration take real coefficients only, the others go on with
the general stencils and BiCGStab.  Against the oracle, through the operator
(before and after a stencil was chosen, and with the FMA stencil asked for) and
over three updates by default, on an even lattice and on an odd one; then real
coefficients on the same solver.

Operator: 1e-13 of the field's scale, as in the other operator tests.  Updates:
the solve ends at a residual of tol |b| a column and A^H stays within a few per
cent of normal, so three leave a few tol."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
REAL = [1.0, 0.9, 1.1, 0.8]
TOL = 1e-12


def coefficients(k):
    c = [complex(v) for v in REAL]
    c[k] += 0.5j
    return c


def field(n, seed):
    rng = np.random.default_rng(seed)
    V = int(np.prod(n))
    return rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))


def check_operator(oracle, n, links, ef, g, c, herm):
    q, an = field(n, 1), field(n, 2)
    fin, fout = NRQCDField(), NRQCDField()
    fin.upload(q, an)
    nrqcd.apply_operator(g, 1.3, c, 1.0, herm, fin, fout)
    oq, oa = fout.download()
    for got, want in ((oq, oracle.cn_apply(n, A, links, ef, 1.3, c, 1.0, int(herm), q)),
                      (oa, oracle.cn_apply(n, A, links, ef, -1.3, np.conj(c), 1.0, int(herm), an))):
        assert np.abs(got - want).max() < 1e-13 * np.abs(q).max()


@pytest.mark.parametrize("n", [(6, 6, 6), (5, 7, 3)])
@pytest.mark.parametrize("k", [0, 1, 2, 3])
def test_one_complex_coefficient(oracle, k, n):
    links, ef = oracle.transverse_box(n, A, 3.0, 1.0, 0.0, 5, identity_links=False)
    c = coefficients(k)
    q, an = oracle.single_point(n, 2), oracle.single_point(n, 3)
    with lattice_ctx(n, A, cn=(1.3, c, 1.0, TOL)):
        g = GaugeConfiguration()
        g.upload(links, ef)
        for herm in (False, True):
            check_operator(oracle, n, links, ef, g, c, herm)
        h = NRQCDField()
        h.InitSinglePoint(2, 3)
        for coeffs in (c, c, c, REAL, c):
            st = h.Update(g, 1.3, coeffs, 1.0)
            assert st["converged"] == 1 and st["max_rel_residual"] <= TOL
            oracle.cn_update(n, A, links, ef, 1.3, coeffs, 1.0, q, an, tol=1e-14)
        gq, ga = h.download()
        for herm in (False, True):
            check_operator(oracle, n, links, ef, g, c, herm)
            check_operator(oracle, n, links, ef, g, REAL, herm)
        if np.prod(n) % 2 == 0:
            nrqcd.SetStencil(nrqcd.STENCIL_FMA)
            check_operator(oracle, n, links, ef, g, c, True)
            check_operator(oracle, n, links, ef, g, REAL, True)
    for got, want in ((gq, q), (ga, an)):
        assert np.linalg.norm(got - want) < 20 * TOL * np.linalg.norm(want)
