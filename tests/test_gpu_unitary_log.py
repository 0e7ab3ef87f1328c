"""The series for the logarithm of a unitary matrix (field strength of the
Crank-Nicolson operator) against the oracle's Jacobi logarithm, on links from
nearly trivial to rough: the series takes matrices whose |sin^2(theta/2)|_F
is at most 3/4, the Jacobi route the others, and rough fields mix both in a
warp.

Tolerance: operator 1e-13 of the field's scale, as in the other operator
tests."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
N = (6, 5, 4)


def rough_links(scale, seed):
    """exp(i scale h) with h traceless hermitian, entries of order one."""
    V = int(np.prod(N))
    rng = np.random.default_rng(seed)
    h = rng.normal(size=(V, 3, 3, 3)) + 1j * rng.normal(size=(V, 3, 3, 3))
    h = (h + h.conj().transpose(0, 1, 3, 2)) / 2
    h -= np.trace(h, axis1=2, axis2=3)[..., None, None] / 3 * np.eye(3)
    w, v = np.linalg.eigh(h)
    u = np.einsum("xdij,xdj,xdkj->xdik", v, np.exp(1j * scale * w), v.conj())
    return np.ascontiguousarray(u.transpose(0, 1, 3, 2)), 0.02 * rng.normal(size=(V, 3, 8))


@pytest.mark.parametrize("scale", [0.0, 1e-9, 0.01, 0.1, 0.2, 0.4, 0.7])
def test_log_matches_jacobi(oracle, scale):
    links, ef = rough_links(scale, 5)
    V = int(np.prod(N))
    rng = np.random.default_rng(1)
    q = rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))
    an = rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))
    M, c = 1.0, [1, 1, 1, 1]
    with lattice_ctx(N, A, cn=(M, c, 1.0, 1e-12)):
        g = GaugeConfiguration()
        g.upload(links, ef)
        fin, fout = NRQCDField(), NRQCDField()
        fin.upload(q, an)
        nrqcd.apply_operator(g, M, c, 1.0, True, fin, fout)
        oq, oa = fout.download()
    size = np.abs(q).max()
    assert np.abs(oq - oracle.cn_apply(N, A, links, ef, M, c, 1.0, 1, q)).max() < 1e-13 * size
    assert np.abs(oa - oracle.cn_apply(N, A, links, ef, -M, c, 1.0, 1, an)).max() < 1e-13 * size
