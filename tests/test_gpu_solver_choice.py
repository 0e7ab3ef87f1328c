"""Which solver the plain form runs: naming the default of the BiCGStab update
leaves the Chebyshev semi-iteration in place and comes back to it from the
two-pass update; beside a forced FMA stencil it selects BiCGStab.  The semi-
iteration applies the operator once a step, BiCGStab twice an iteration."""
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)


def test_default_update_named(oracle):
    n = (8, 8, 8)
    links, ef = oracle.transverse_box(n, A, 2.0, 1.0, 0.0, 4, identity_links=False)
    with lattice_ctx(n, A, cn=(1.0, [1, 1, 1, 1], 1.0, 1e-12)):
        nrqcd.SetTrueResidual(True)
        g = GaugeConfiguration()
        g.upload(links, ef)

        def first():
            h = NRQCDField()
            h.InitSinglePoint(1, 1)
            st = h.Update(g, 1.0, [1, 1, 1, 1], 1.0)
            assert st["converged"] == 1 and st["max_rel_residual"] <= 1e-12
            return st["iterations"], st["matvecs"]

        default = first()
        nrqcd.SetMergedUpdate(True)
        assert first() == default
        nrqcd.SetMergedUpdate(False)
        its, applies = first()
        assert applies >= 2 * its and its < default[0]
        nrqcd.SetMergedUpdate(True)
        assert first() == default
        nrqcd.SetStencil(nrqcd.STENCIL_FMA)
        its, applies = first()
        assert applies >= 2 * its and its < default[0]
        nrqcd.SetStencil(None)
        assert first() == default
