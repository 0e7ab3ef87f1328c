"""The first updates of a batch, while its fields' histories fill, against plain
FP64 solves at 1e-13.  Passes then aim 0.05 tol |b| and |A^H^-1| <= 1, so k
updates leave at most 0.05 k tol of a propagator and the little that FP32 passes
of gains up to 1e6 add; 0.125 k tol is asked for."""
import numpy as np
import pytest

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from nrqcd_b200.batch import CNBatch
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)
TOL = 1e-10
C = [1, 1, 1, 1]
SITES, MASSES = (1, 100, 333), (1.0, 1.5)


@pytest.mark.parametrize("n", [(12, 10, 8), (24, 24, 24)])
def test_first_updates(oracle, n):
    links, ef = oracle.transverse_box(n, A, 2.0, 1.0, 0.0, 4, identity_links=False)
    got, ref = [], []
    with lattice_ctx(n, A):
        g = GaugeConfiguration()
        g.upload(links, ef)
        fields, masses = [], []
        for m in MASSES:
            for s in SITES:
                fields.append(NRQCDField())
                fields[-1].InitSinglePoint(s, s)
                masses.append(m)
        b = CNBatch(fields, masses, TOL)
        for _ in range(3):
            assert b.Update(g, C, 1.0)["converged"] == 1
            got.append([np.stack(f.download()) for f in fields])
            g.Update(1.0)
        b.Destructor()
    for m in MASSES:
        with lattice_ctx(n, A, cn=(m, C, 1.0, 1e-13)):
            nrqcd.SetTrueResidual(True)
            g = GaugeConfiguration()
            g.upload(links, ef)
            fields = []
            for s in SITES:
                fields.append(NRQCDField())
                fields[-1].InitSinglePoint(s, s)
            ref.append([])
            for _ in range(3):
                for f in fields:
                    assert f.Update(g, m, C, 1.0)["converged"] == 1
                ref[-1].append([np.stack(f.download()) for f in fields])
                g.Update(1.0)
    for k in range(3):
        want = ref[0][k] + ref[1][k]
        for x, y in zip(got[k], want):
            assert np.linalg.norm(x - y) <= 0.125 * (k + 1) * TOL * np.linalg.norm(y), k + 1
