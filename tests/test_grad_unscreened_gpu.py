"""A negative Schwarz threshold skips no quartet: the gradient equals that of
threshold zero."""
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutint", [-1.0, -0.5])
def test_negative_threshold_keeps_every_quartet(cutint):
    g = MolGpu(B.small_molecule(3, seed=5))
    D = torch.from_numpy(B.density_factor(g.nbf, 5, 5)).cuda()
    D = D @ D.t()
    got = g.drvg1(D, cutint=cutint)
    want = g.drvg1(D, cutint=0.0)
    # (atomic sums: rounding only)
    assert float((got - want).abs().max()) <= 1e-12 * float(want.abs().max())
    assert len(g.grad_plan_info()) > 0
