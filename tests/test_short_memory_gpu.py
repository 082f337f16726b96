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


@pytest.mark.parametrize("natom,thrcom,r", [(6, 1e-7, 9), (46, 0.3, 17)])
def test_jk_workspaces_shrink(natom, thrcom, r):
    """J/K calls whose workspace is refused again and again run with fewer vectors
    per launch: the FP64 path against the products of the unpacked vectors (bars
    of its tests), the mixed one against it, until nothing smaller is left."""
    from tests.test_jk64_gpu import _reference
    mol = B.make_molecule("shrink", natom, [("3s2p1d", natom)], 6)
    g = MolGpu(mol)
    g.cho_drv(thrcom=thrcom)
    C = _density(g, r)
    Jr, Kr, tj, tk = _reference(g, C)
    for prec, bars in ((MolGpu.PREC_FP64, (tj, tk)),
                       (MolGpu.PREC_MIXED, (1e-13 * float(Jr.abs().max()) + tj, 1e-10 * float(Kr.abs().max()) + tk))):
        done = 0
        for tries in range(1, 40):
            g2 = MolGpu(mol)
            g2.cho_drv(thrcom=thrcom)
            g2.cho_jk(_density(g, 1))  # the tables that belong to the vectors are there
            try:
                # (each request is made twice)
                with refuse(0, 2 * tries) as rf:
                    J, K = g2.cho_jk(C, precision=prec)
            except MolGpuError:
                break
            if rf.failed == 2 * tries:
                done += 1
                assert float((J - Jr).abs().max()) <= bars[0]
                assert float((K - Kr).abs().max()) <= bars[1]
        assert done >= 2  # (how many steps there are depends on the number of vectors)
        assert g2.cho_jk(C, precision=prec)[1].any()


def test_gradient_after_a_plan_that_could_not_be_made():
    """A re-plan (another threshold) that is refused memory leaves no half-made plan
    to a call with the old threshold."""
    g = MolGpu(B.small_molecule(3, seed=5))
    D = _density(g, 5)
    D = D @ D.t()
    want = g.drvg1(D, cutint=1e-12)
    for skip in range(3):
        with pytest.raises(MolGpuError, match="rc=2"), refuse(skip):
            g.drvg1(D, cutint=1e-10)
        got = g.drvg1(D, cutint=1e-12)
        # (atomic sums: rounding only)
        assert float((got - want).abs().max()) <= 1e-12 * float(want.abs().max())
