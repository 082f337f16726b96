"""A decomposition on another stream than the calls that still read the vectors
it replaces: FP64 J/K and vector copies queued behind a delay on one stream keep
their vectors, although the next decomposition (other pivots, the same AO-pair
list) reuses their storage on another stream."""
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu

pytestmark = pytest.mark.gpu
DELAY = 400_000_000  # clocks, some 0.2 s


def test_replaced_vectors_outlive_their_readers():
    g = MolGpu(B.make_molecule("streams", 6, [("3s2p1d", 6)], 4))
    g.cho_drv(thrcom=1e-5)
    C = torch.from_numpy(B.density_factor(g.nbf, 9, 9)).cuda()
    J0, K0 = g.cho_jk(C)
    L0 = g.cho_vectors()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(DELAY)
        J1, K1 = g.cho_jk(C)
        L1 = g.cho_vectors()
    with torch.cuda.stream(s2):
        g.cho_drv(thrcom=1e-5, span=0.9)
    torch.cuda.synchronize()
    assert not torch.equal(g.cho_vectors()[:L0.shape[0]], L0[:g.cho_info()["M"]])
    assert torch.equal(J1, J0) and torch.equal(K1, K0) and torch.equal(L1, L0)


def test_first_fp64_jk_after_a_decomposition_only_queues():
    """FP64 J/K calls queue their kernels and return, the first call over new vectors
    included: behind a delay on the same stream the call comes back before the
    delay has ended."""
    g = MolGpu(B.make_molecule("queue", 6, [("3s2p1d", 6)], 4))
    g.cho_drv(thrcom=1e-5)
    C = torch.from_numpy(B.density_factor(g.nbf, 9, 9)).cuda()
    J0, K0 = g.cho_jk(C)  # (the workspace is there)
    g.cho_drv(thrcom=1e-5)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        done = torch.cuda.Event()
        torch.cuda._sleep(DELAY)
        done.record()
        J1, K1 = g.cho_jk(C)
        pending = not done.query()
    torch.cuda.synchronize()
    assert pending
    assert torch.equal(J1, J0) and torch.equal(K1, K0)
