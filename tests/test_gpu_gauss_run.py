"""The Gauss projection's two forms at their edges: one launch of many sweeps
on lattices of up to 100 sites a multiprocessor, one thread per link and ten
sites a warp, and two launches a sweep above.  Twenty sweeps against the
oracle: a sweep rounds a handful of times at the field's size, so 1e-13 of it
leaves a factor of five."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration
from nrqcd_b200._capi import NrqcdError
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.1, 1.0, 0.9, 1.1)


# one full warp and a ragged one; warps that end inside a row; just below and
# above 100 x 148 sites
@pytest.mark.parametrize("n", [(5, 2, 2), (3, 3, 3), (7, 11, 2), (25, 24, 24), (25, 25, 24)])
def test_twenty_sweeps(oracle, n):
    rng = np.random.default_rng(4)
    links, ef = oracle.transverse_box(n, A, 2.0, 1.0, 0.0, 9, identity_links=False)
    ef = ef + 0.02 * rng.standard_normal(ef.shape)
    with lattice_ctx(n, A):
        g = GaugeConfiguration()
        g.upload(links, ef)
        with pytest.raises(NrqcdError):
            g.GaussProjection(1e-9, max_sweeps=20)
        _, got = g.download()
    want, l = ef.copy(), links.copy()
    assert oracle.gauss_project(n, A, l, want, tol=1e-9, max_sweeps=20) == 20
    assert np.abs(got - want).max() < 1e-13 * np.abs(want).max()
