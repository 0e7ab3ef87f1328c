"""The streaming observables at block edges: norms of either species alone
and together, and the meson correlators (plain and _gconjg), on random
propagators whose volumes straddle the 128-site blocks, against the oracle.

Tolerance: sums of V*36 products of order one in a different order, relative
error at most about sqrt(36 V) eps (1e-14 at the largest); 1e-12 relative to
the largest term's scale V leaves two digits."""
import ctypes

import numpy as np
import pytest

from nrqcd_b200 import NRQCDField, _capi
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)


@pytest.mark.parametrize("n", [(1, 1, 1), (127, 1, 1), (8, 4, 4), (43, 3, 1), (16, 16, 9)])
def test_norms_and_correlators_at_block_edges(oracle, n):
    V = int(np.prod(n))
    rng = np.random.default_rng(V)
    q = rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))
    an = rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))
    with lattice_ctx(n, A):
        h = NRQCDField()
        h.upload(q, an)
        both = (ctypes.c_double(), ctypes.c_double())
        _capi.check(_capi.load().nrq_heavy_norms(h.handle, *(ctypes.byref(v) for v in both)))
        alone = (h.GetNorm_Quark(), h.GetNorm_AntiQ())
        plain, conj = h.GetMesoncorrelators(), h.GetMesoncorrelators_gconjg()
    for got, one, field in zip(both, alone, (q, an)):
        assert got.value == one
        assert abs(one - oracle.heavy_norm(n, field)) <= 1e-12 * one
    for got, want in ((plain, oracle.meson_correlators(n, q, an)), (conj, oracle.meson_correlators_gconjg(n, q, an))):
        for k in want:
            assert abs(got[k] - want[k]) <= 1e-12 * 36 * V, k
