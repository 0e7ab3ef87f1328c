"""The Coulomb gauge fixing's two forms at their edges: extents up to 32 with
transforms of their own, odd, prime and tiny ones among them, and one of 33
through the library's.  Five iterations against the oracle: each adds a few
roundings of order-one links, so 1e-12 leaves a factor of a hundred."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.2, 0.9)


@pytest.mark.parametrize("n", [(2, 3, 2), (7, 4, 5), (32, 3, 2), (3, 31, 2), (2, 2, 32), (33, 3, 2)])
def test_five_iterations(oracle, n):
    links, ef = oracle.transverse_box(n, A, 1.0, 1.0, 0.5, 3, identity_links=False)
    for _ in range(10):
        oracle.gauge_update(n, A, links, ef, 1.0)
    with lattice_ctx(n, A):
        g = GaugeConfiguration()
        g.upload(links, ef)
        it, dev = g.CoulombGaugefixing(1e-30, 0.08, 5, verbose=False)
        got, _ = g.download()
    it_ref, dev_ref = oracle.coulomb_gaugefix(n, A, links, tol=1e-30, alpha=0.08, max_iterations=5)
    assert it == it_ref == 6
    assert np.allclose(dev, dev_ref, rtol=1e-10, atol=1e-14)
    assert np.abs(got - links).max() < 1e-12
