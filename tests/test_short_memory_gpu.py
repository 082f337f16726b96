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


def test_kept_memory_gives_way():
    """One refusal at every allocation of a second decomposition (more qualified
    columns, so that its buffers grow), then of the calls after it: what the handle
    keeps is freed, the request repeated, and the results are the same."""
    mol = B.make_molecule("keep", 6, [("3s2p1d", 6)], 4)
    g0 = MolGpu(mol)
    g0.cho_drv(thrcom=1e-6)
    L0, C = g0.cho_vectors(), _density(g0, 7)
    jk0 = [g0.cho_jk(C, precision=p) for p in (MolGpu.PREC_FP64, MolGpu.PREC_MIXED)]
    grad0 = g0.drvg1(C @ C.t())
    calls = [lambda g: g.cho_jk(C, precision=MolGpu.PREC_FP64), lambda g: g.cho_jk(C, precision=MolGpu.PREC_MIXED),
             lambda g: (g.drvg1(C @ C.t()),)]
    wants = jk0 + [(grad0,)]
    for skip in range(8):
        g = MolGpu(mol)
        g.cho_drv(thrcom=1e-6, maxqual=2)
        with refuse(skip, 1) as r:
            g.cho_drv(thrcom=1e-6)
        assert torch.equal(g.cho_vectors(), L0)
        for call, want in zip(calls, wants):
            with refuse(skip, 1):
                got = call(g)
            for a, b in zip(got, want):
                # (the gradient and the mixed exchange add with atomics: rounding only)
                assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())
        assert skip or r.failed == 1
