"""The history that a precision update leaves, x - (2b - psi) stored by the last
launch of a pass of the spin-structured step (or by a pass of one step, or by a
launch of its own where the start was good enough), against the register-tiled
step's, which always takes the latter: the next updates start from the same
residuals.  The passes' corrections agree to the rounding of FP32 numbers,
which the extrapolation from four vectors amplifies 15 times: 15 x 6e-8 of the
vectors' size a start, of which 2 % of a start's residual leaves room down to
1e-4 of that size."""
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)


@pytest.mark.parametrize("mass,tol", [(1.0, 1e-8), (1.0, 1e-5), (1.0, 1e-3), (10.0, 1e-8), (10.0, 1e-6), (10.0, 1e-5)])
def test_starts_agree(oracle, mass, tol):
    n = (10, 6, 4)
    links, ef = oracle.transverse_box(n, A, 2.0, 1.0, 0.0, 4, identity_links=False)
    starts = {}
    for cheb in (nrqcd.CHEB_BLOCKS, nrqcd.CHEB_REGISTER):
        with lattice_ctx(n, A, cn=(mass, [1, 1, 1, 1], 1.0, tol, 10000, nrqcd.FORM_PRECISION)):
            nrqcd.SetChebStencil(cheb)
            g = GaugeConfiguration()
            g.upload(links, ef)
            h = NRQCDField()
            h.InitSinglePoint(1, 1)
            starts[cheb] = []
            for _ in range(6):
                st = h.Update(g, mass, [1, 1, 1, 1], 1.0)
                assert st["converged"] == 1
                starts[cheb].append((st["initial_rel_residual"], st["iterations"]))
                g.Update(1.0)
    for (x, i), (y, j) in zip(*starts.values()):
        assert abs(x - y) <= 0.02 * y and i == j, starts
