"""Mixed J/K with several blocks of vectors per launch: systems whose blocks go
sixteen, four and two to a launch, with a short last block and fewer blocks than
a launch takes, one and three densities of uneven rank, against the FP64 path
with the bars of the mixed path (K within 1e-10, J within 1e-13 of the largest
element)."""
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natom,thrcom", [(2, 1e-3), (6, 1e-7), (14, 1e-6), (22, 1e-4)])
def test_mixed_against_fp64(natom, thrcom):
    g = MolGpu(B.make_molecule("groups", natom, [("3s2p1d", natom)], 6))
    g.cho_drv(thrcom=thrcom)
    Cs = [torch.from_numpy(B.density_factor(g.nbf, r, 70 + r)).cuda() for r in (1, 9, max(2, g.nbf // 6))]
    ref = g.cho_jk_batch(Cs, precision=MolGpu.PREC_FP64)
    one = g.cho_jk(Cs[-1], precision=MolGpu.PREC_MIXED)
    for got, want in list(zip(g.cho_jk_batch(Cs, precision=MolGpu.PREC_MIXED), ref)) + [(one, ref[-1])]:
        for a, b, bar in ((got[0], want[0], 1e-13), (got[1], want[1], 1e-10)):
            assert float((a - b).abs().max()) < bar * float(b.abs().max())
            assert torch.equal(a, a.t())
