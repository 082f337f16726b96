"""J/K over a decomposition without vectors: a threshold above the largest
diagonal (the reduced set is empty after the first look) and one so large that
the initial screening leaves no AO pair at all.  Both precisions give zeros and
add nothing to a Fock matrix; a decomposition that fails before its first vector
leaves none behind."""
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu, MolGpuError

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    return MolGpu(B.small_molecule(3, seed=5))


@pytest.mark.parametrize("precision", [MolGpu.PREC_FP64, MolGpu.PREC_MIXED, MolGpu.PREC_SLICED(4)])
@pytest.mark.parametrize("factor", [2.0, 1e9])
def test_zero_vectors_give_zero_matrices(g, factor, precision):
    g.cho_drv(thrcom=1e-6)
    top = float(g.cho_diag().max())
    info = g.cho_drv(thrcom=factor * max(top, 1.0))
    assert info["M"] == 0 and (info["nrs"] == 0) == (factor > 1e8)
    Cs = [torch.from_numpy(B.density_factor(g.nbf, r, r)).cuda() for r in (1, 5)]
    for J, K in g.cho_jk_batch(Cs, precision=precision) + [g.cho_jk(Cs[0], precision=precision)]:
        assert not J.any() and not K.any()
    F = torch.randn(g.nbf, g.nbf, dtype=torch.float64, device="cuda")
    F0 = F.clone()
    g.choscf_lk(Cs[1] @ Cs[1].t(), 0.5, F, precision=precision)
    assert torch.equal(F, F0)


def test_failed_decomposition_without_vectors_is_dropped(g):
    g.cho_drv(thrcom=1e-6)
    with pytest.raises(MolGpuError, match="rc=2"):
        g.cho_drv(thrcom=1e-6, maxvec=1, maxqual=100)
    C = torch.from_numpy(B.density_factor(g.nbf, 3, 3)).cuda()
    with pytest.raises(MolGpuError, match="no Cholesky vectors"):
        g.cho_jk(C)
    g.cho_drv(thrcom=1e-6)
    assert g.cho_jk(C)[1].any()
