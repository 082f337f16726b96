"""Cholesky passes with many pivots (k_cho_subtr / k_cho_compvec in cholesky.cu):
general contractions whose passes take up to 57 pivots from one shell pair, so
that a pass runs in more than one launch, and a repeated decomposition that
reuses the storage of the first, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu

pytestmark = pytest.mark.gpu


def test_passes_with_more_than_32_pivots():
    mol = B.make_molecule("big", 2, [("4s3p2d", 2)], 2)
    ref = O.Oracle(mol).cholesky(thrcom=1e-6)
    assert np.bincount(ref["pass_of"]).max() > 32
    g = MolGpu(mol)
    first = None
    for _ in range(2):
        info = g.cho_drv(thrcom=1e-6)
        piv, pas = g.cho_pivots()
        assert info["M"] == ref["M"]
        assert np.array_equal(piv, ref["piv"]) and np.array_equal(pas, ref["pass_of"])
        L = g.cho_vectors().cpu().numpy().T
        # the bar of the decomposition tests
        assert np.abs(L - ref["L"]).max() < 1e-9
        assert first is None or np.array_equal(L, first)
        first = L


@pytest.mark.parametrize("n,rank", [(1, 1), (33, 7), (1500, 40), (10001, 3)])
def test_cd_incore_sizes(n, rank):
    """In-core decomposition on one row, a partial warp, more rows than threads
    and more than the staged pivot row holds; equal diagonals (the running-maximum
    rule picks the first) among them.  Reconstruction within the threshold plus
    rounding (n + rank products of size <= max diagonal)."""
    import torch
    rng = np.random.default_rng(n)
    V = rng.standard_normal((n, rank))
    V[: n // 2] /= np.linalg.norm(V[: n // 2], axis=1, keepdims=True)  # diagonals equal to rounding
    g = MolGpu(B.small_molecule(2, mix=[("2s1p", 2)]))
    X = torch.from_numpy(V).cuda()
    X = X @ X.t()
    top = float(X.diagonal().max())
    W, irc = g.cd_incore(X, thr=1e-8 * top)
    assert irc == 0 and W.shape[1] == min(n, rank)
    assert float((X - W @ W.t()).abs().max()) <= 1e-8 * top + 4 * (n + rank) * 2.0 ** -53 * top
