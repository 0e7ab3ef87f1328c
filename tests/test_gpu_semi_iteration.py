"""The plain solve's Chebyshev semi-iteration against two-pass BiCGStab
(SetMergedUpdate selects BiCGStab) at its edges: odd and ragged lattices of one
partial unit of 32 sites and more, a unit boundary, and a step so large for its
mass that the enclosure asks for more steps than the coefficient table holds and
the solve falls back to BiCGStab by itself.

Both end at a residual of at most tol |b| a column and |A^H^-1| <= 1, so the
propagators differ by at most 2 tol |b| a step, |b| <= |1 + i tau lambda| |psi|
with lambda up to 6.6 / mass (the free spectrum's 6 / mass and a tenth for the
fields); the steps preserve norms, so three leave 6 tol |1 + i tau lambda|."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _run(oracle, n, a, mass, bicgstab):
    links, ef = oracle.transverse_box(n, a, 3.0, 1.0, 0.0, 5, identity_links=False)
    with lattice_ctx(n, a, cn=(mass, [1, 1, 1, 1], 1.0, TOL)):
        if bicgstab:
            nrqcd.SetMergedUpdate(False)
        g = GaugeConfiguration()
        g.upload(links, ef)
        h = NRQCDField()
        h.InitSinglePoint(1, 1)
        stats = [h.Update(g, mass, [1, 1, 1, 1], 1.0) for _ in range(3)]
        return np.stack(h.download()), stats


@pytest.mark.parametrize("n,a0,mass", [((3, 3, 3), 0.05, 1.0), ((5, 7, 3), 0.05, 2.5), ((8, 4, 1), 0.05, 1.0),
                                       ((11, 3, 1), 0.05, 1.0), ((32, 8, 8), 0.1, 1.0), ((5, 4, 6), 0.5, 0.5),
                                       ((5, 4, 6), 1.0, 0.5)])
def test_semi_iteration_matches_bicgstab(oracle, n, a0, mass):
    a = (a0, 1.0, 1.0, 1.0)
    x, sx = _run(oracle, n, a, mass, False)
    y, sy = _run(oracle, n, a, mass, True)
    for s in sx + sy:
        assert s["converged"] == 1 and s["max_rel_residual"] <= TOL
    # per species and column: (2, V, column, row)
    x, y = (np.moveaxis(f.reshape(2, -1, 6, 6), 1, 3).reshape(12, -1) for f in (x, y))
    diff = np.linalg.norm(x - y, axis=1) / np.linalg.norm(y, axis=1)
    assert diff.max() < 6 * TOL * np.hypot(1.0, 0.5 * a0 * 6.6 / mass), diff
