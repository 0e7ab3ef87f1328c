"""The per-update operator takes memory only where a kernel that reads it runs:
a precision solver on the register-tiled kernels adds the seven real planes of
its spectral enclosure and a few rows (56 B a site), not the operator's 1.5 KB
(FP64) or 0.8 KB (FP32); a plain solver adds the operator and those, and no
tensor-core blocks (3.4 KB), also after a timed choice that they lose.
Allocations come in pages of 2 MB: one for each."""
import pytest
import torch

from nrqcd_b200 import GaugeConfiguration, NRQCDField, nrqcd
from tests.gpu_util import lattice_ctx

pytestmark = pytest.mark.gpu

A = (0.05, 1.0, 1.0, 1.0)


@pytest.mark.parametrize("n", [(40, 32, 32), (41, 31, 33)])
def test_register_kernels_need_no_operator(n):
    V = n[0] * n[1] * n[2]
    with lattice_ctx(n, A, cn=(1.0, [1, 1, 1, 1], 1.0, 1e-10, 10000, nrqcd.FORM_PRECISION)):
        nrqcd.SetStencil(nrqcd.STENCIL_REGISTER)
        nrqcd.SetChebStencil(nrqcd.CHEB_REGISTER)
        nrqcd.SetHistoryGuess(False)
        g = GaugeConfiguration()
        g.ColdInit()
        h = NRQCDField()
        h.InitSinglePoint(1, 1)
        before = torch.cuda.mem_get_info()[0]
        assert h.Update(g, 1.0, [1, 1, 1, 1], 1.0)["converged"] == 1
        used = before - torch.cuda.mem_get_info()[0]
        assert used <= 56 * V + 4 * 2 ** 21, used / V


@pytest.mark.parametrize("timed", [False, True])
def test_plain_solver_keeps_no_blocks(timed):
    n = (40, 32, 32)
    V = n[0] * n[1] * n[2]
    with lattice_ctx(n, A, cn=(1.0, [1, 1, 1, 1], 1.0, 1e-12)):
        if timed:
            nrqcd.SetStencil(None)
        nrqcd.SetHistoryGuess(False)
        g = GaugeConfiguration()
        g.ColdInit()
        h = NRQCDField()
        h.InitSinglePoint(1, 1)
        before = torch.cuda.mem_get_info()[0]
        assert h.Update(g, 1.0, [1, 1, 1, 1], 1.0)["converged"] == 1
        used = before - torch.cuda.mem_get_info()[0]
        which, ms = nrqcd.StencilInfo()
        assert which == nrqcd.STENCIL_FMA and (ms > 0).all() == timed
        assert used <= (1512 + 56) * V + 8 * 2 ** 21, used / V
