"""Links that are not unitary: the logarithm's series holds for unitary
matrices alone, and the reference's eigenphases (src/matrixoperations.f90:
327-531) for any.  Against the oracle: the transverse correlators with links off
by 1e-3 in every entry and by the 1e-7 of FP32 storage, and the Crank-Nicolson
operator with links times 1.001, smooth and rough (a plaquette that is not
normal gives another logarithm in the other orientation, which the reference
takes for one of the three planes).

The Gauss projection in the generators' coordinates drops the trace of U^+ E U,
so that links that are not unitary take its matrix form.

Tolerances as in the other tests of these: 1e-13 of the field's scale and 1e-11
of the largest correlator."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from nrqcd_b200._capi import NrqcdError
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
N = (6, 5, 4)
V = int(np.prod(N))


def links_off_by(scale, defect, factor=1.0):
    """factor exp(i scale h) plus noise of size `defect` (None: rounded to FP32)."""
    rng = np.random.default_rng(5)
    h = rng.normal(size=(V, 3, 3, 3)) + 1j * rng.normal(size=(V, 3, 3, 3))
    h = (h + h.conj().transpose(0, 1, 3, 2)) / 2
    h -= np.trace(h, axis1=2, axis2=3)[..., None, None] / 3 * np.eye(3)
    w, v = np.linalg.eigh(h)
    u = factor * np.einsum("xdij,xdj,xdkj->xdik", v, np.exp(1j * scale * w), v.conj())
    if defect is None:
        u = u.astype(np.complex64).astype(np.complex128)
    else:
        u = u + defect * (rng.normal(size=u.shape) + 1j * rng.normal(size=u.shape))
    return np.ascontiguousarray(u.transpose(0, 1, 3, 2)), 0.02 * rng.normal(size=(V, 3, 8))


@pytest.mark.parametrize("scale", [0.05, 0.2, 0.4])
def test_operator(oracle, scale):
    links, ef = links_off_by(scale, 0.0, 1.001)
    rng = np.random.default_rng(1)
    q = rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))
    with lattice_ctx(N, A, cn=(1.0, [1, 1, 1, 1], 1.0, 1e-12)):
        nrqcd.SetStencil(nrqcd.STENCIL_FMA)
        g = GaugeConfiguration()
        g.upload(links, ef)
        fin, fout = NRQCDField(), NRQCDField()
        fin.upload(q, q)
        nrqcd.apply_operator(g, 1.0, [1, 1, 1, 1], 1.0, True, fin, fout)
        oq, oa = fout.download()
    for got, mass in ((oq, 1.0), (oa, -1.0)):
        want = oracle.cn_apply(N, A, links, ef, mass, [1, 1, 1, 1], 1.0, 1, q)
        assert np.abs(got - want).max() < 1e-13 * np.abs(q).max()


@pytest.mark.parametrize("defect", [1e-3, None])
def test_transverse_correlators(oracle, defect):
    links, ef = links_off_by(0.1, defect)
    with lattice_ctx(N, A):
        g = GaugeConfiguration()
        g.upload(links, ef)
        aa, ee, _ = g.GetTransverseCorrelators()
    raa, ree, _ = oracle.transverse_correlators(N, A, links, ef)
    assert np.abs(aa - raa).max() < 1e-11 * np.abs(raa).max()
    assert np.abs(ee - ree).max() < 1e-11 * np.abs(ree).max()


@pytest.mark.parametrize("defect,factor", [(1e-3, 1.0), (None, 1.0), (0.0, 1.001)])
def test_gauss_projection(oracle, defect, factor):
    links, ef = links_off_by(0.2, defect, factor)
    a = (0.1, 1.0, 0.9, 1.1)
    with lattice_ctx(N, a):
        g = GaugeConfiguration()
        g.upload(links, ef)
        with pytest.raises(NrqcdError):
            g.GaussProjection(1e-9, max_sweeps=20)
        _, got = g.download()
    want, l = ef.copy(), links.copy()
    assert oracle.gauss_project(N, a, l, want, tol=1e-9, max_sweeps=20) == 20
    assert np.abs(got - want).max() < 1e-13 * np.abs(want).max()
