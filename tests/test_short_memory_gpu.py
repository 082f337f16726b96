"""Device memory that runs short: allocations refused on request
(mg_test_fail_allocations) at the points where a call asks for memory."""
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu, MolGpuError, lib

pytestmark = pytest.mark.gpu
ALL = 1 << 20


class refuse:
    """Within the block, `skip` allocations of the library proceed and `count` more fail."""

    def __init__(self, skip, count=ALL):
        self.skip, self.count = skip, count

    def __enter__(self):
        lib().mg_test_fail_allocations(self.skip, self.count)
        return self

    def __exit__(self, *exc):
        self.failed = self.count - lib().mg_test_fail_allocations(0, 0)


def _density(g, r):
    return torch.from_numpy(B.density_factor(g.nbf, r, r)).cuda()


def test_a_refused_call_leaves_no_error_behind():
    g = MolGpu(B.small_molecule(3, seed=5))
    g.cho_drv(thrcom=1e-6)
    C = _density(g, 5)
    for prec in (MolGpu.PREC_FP64, MolGpu.PREC_MIXED):
        with pytest.raises(MolGpuError, match="rc=2"), refuse(0):
            g.cho_jk(C, precision=prec)
        assert g.cho_jk(C, precision=prec)[1].any()
