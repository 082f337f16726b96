"""The 8-bit sliced half-transform over more than one K chunk (oz_gemm.cuh reads
its accumulators out every 4096 K elements): the row maxima that scale the slices
of X must be those of the whole sums, not of the last chunk's share.

Bars at 8 slices: an operand's dropped tail is below 2^-63 of its power-of-two
scale (below twice the row's largest element), the products left out (diagonals
8 and above) below 9 2^-62, the FP64 recombination and the reference's own sum
below 2^-53 each, all per product: 4 N (2 2^-53 + 9 2^-62) max|row| max|column|
over N products."""
import numpy as np
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu
from tests.test_jk_gpu import _selftest

pytestmark = pytest.mark.gpu
PER_PRODUCT = 4.0 * (2.0 * 2.0 ** -53 + 9.0 * 2.0 ** -62)


@pytest.mark.parametrize("ld", [4096, 4224])
def test_row_maxima_over_k_chunks(ld):
    g = MolGpu(B.small_molecule(2, mix=[("2s1p", 2)]))
    rng = np.random.default_rng(ld)
    A = rng.standard_normal((ld, ld))
    Bm = rng.standard_normal((5, ld))
    A[:, -128:] *= 1e-3  # the last chunk adds little to any sum
    X, K = _selftest(g, A, Bm, 8)
    Xe = (torch.from_numpy(A).cuda() @ torch.from_numpy(Bm).cuda().t()).cpu().numpy()
    assert np.abs(X - Xe).max() <= PER_PRODUCT * ld * np.abs(A).max() * np.abs(Bm).max()
    Ke = X @ X.T
    lo = np.tril_indices(ld)
    assert np.abs(K[lo] - Ke[lo]).max() <= PER_PRODUCT * 5 * np.abs(X).max() ** 2
