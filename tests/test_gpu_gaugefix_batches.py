"""The gauge fixing on short extents queues its iterations in batches (one, eight,
then as many as the decay asks for): counts, deviations and links against the
oracle where it ends in the first, at a batch's edge, inside a later one, and at
the iteration limit.  Links to 1e-11 and deviations to 1e-9, as the gauge
fixing's other tests hold them."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
N = (6, 5, 4)


@pytest.fixture(scope="module")
def fixed(oracle):
    links, ef = oracle.transverse_box(N, A, 1.0, 1.0, 0.5, 3, identity_links=False)
    for _ in range(10):
        oracle.gauge_update(N, A, links, ef, 1.0)
    _, dev = oracle.coulomb_gaugefix(N, A, links.copy(), tol=1e-30, alpha=0.08, max_iterations=45)
    return links, ef, dev


@pytest.mark.parametrize("count,limit", [(1, 100), (2, 100), (9, 100), (10, 100), (16, 100), (0, 9), (0, 10), (0, 1)])
def test_counts(oracle, fixed, count, limit):
    links, ef, dev = fixed
    # met by iteration `count` (0: by none within the limit)
    tol = dev[count - 1] * (1 + 1e-6) if count else 1e-30
    want = links.copy()
    it_ref, dev_ref = oracle.coulomb_gaugefix(N, A, want, tol=tol, alpha=0.08, max_iterations=limit)
    assert it_ref == (count or limit + 1)
    with lattice_ctx(N, A):
        g = GaugeConfiguration()
        g.upload(links, ef)
        it, d = g.CoulombGaugefixing(tol, 0.08, limit, verbose=False)
        got, _ = g.download()
    assert it == it_ref
    assert np.allclose(d, dev_ref, rtol=1e-9, atol=1e-14)
    assert np.abs(got - want).max() < 1e-11
    if count == 1:
        assert np.array_equal(got, links)
