"""The precision form's propagator against a plain FP64 solve, at the larger of
its two production sizes and over enough updates for its history to fill and
its steady state to show.

An update ends at a predicted residual of at most 0.1 tol |b|, or where the
prediction cannot be trusted at a measured one; with the rounding of the FP32
passes (4e-8 of the residual they start from, at most 3e-4) that is at most
0.25 tol, and |A^H^-1| <= 1, so k updates leave at most 0.25 k tol of the
propagator beside the plain solve's 1e-13 an update.  The errors of successive
updates are not aligned; half of it is asked for.  The worst element against
the field's rms: the error lives on the (2k + 1)^3 sites or fewer that the
source has reached, so its rms there is sqrt(V / (2k + 1)^3) times that of the
whole lattice; a factor of 15 above that covers its concentration near the
source."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
TOL = 1e-10


def _run(n, form, tol, after):
    with lattice_ctx(n, A, cn=(1.0, [1, 1, 1, 1], 1.0, tol, 10000, form)):
        if form == nrqcd.FORM_PLAIN_FP64:
            nrqcd.SetTrueResidual(True)
        g = GaugeConfiguration()
        g.TransversePolarisedOccupiedInit_Box(0.5, 1.0, 0.0, RandomSeed=3, identity_links=True)
        h = NRQCDField()
        h.InitSinglePoint(1, 1)
        out = []
        for k in range(1, max(after) + 1):
            st = h.Update(g, 1.0, [1, 1, 1, 1], 1.0)
            assert st["converged"] == 1 and st["max_rel_residual"] <= tol
            g.Update(1.0)
            if k in after:
                out.append(np.stack(h.download()))
        return out


@pytest.mark.parametrize("n", [(20, 18, 16), (96, 96, 96)])
def test_propagator_over_eight_updates(n):
    after = (3, 4, 8)
    got = _run(n, nrqcd.FORM_PRECISION, TOL, after)
    ref = _run(n, nrqcd.FORM_PLAIN_FP64, 1e-13, after)
    V = float(np.prod(n))
    for k, x, y in zip(after, got, ref):
        e = x - y
        norm, size = np.linalg.norm(e), np.linalg.norm(y)
        assert norm <= 0.125 * k * TOL * size, (k, norm / size)
        rms = size / np.sqrt(y.size)
        reached = min(V, (2 * k + 1) ** 3)
        assert np.abs(e).max() <= 15 * np.sqrt(V / reached) * 0.125 * k * TOL * rms, (k, np.abs(e).max() / rms)
