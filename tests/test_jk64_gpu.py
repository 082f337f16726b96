"""FP64 J/K kernels (jk64.cu, coulomb.cuh) at the edges of their tiles: 64-row
tiles of the exchange product with remainders, column counts around
the 8- and 64-column steps of the half-transform, one vector block and several,
against torch products of the unpacked vectors.

Bars: a sum of N products in FP64, in any order, is within N 2^-53 of its exact
value relative to the sum of the absolute products; both sides carry that
error, so they agree within 2 N 2^-53 of that sum."""
import numpy as np
import pytest
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _reference(g, C):
    L = g.cho_vectors()
    a, b, _ = (torch.from_numpy(x.astype(np.int64)).cuda() for x in g.cho_rs_list())
    n, M = g.nbf, L.shape[0]
    D = C @ C.t()
    w = torch.where(a == b, 1.0, 2.0).double()
    dw = w * D[a, b]
    J = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    jrs = L.t() @ (L @ dw)
    J[a, b] = jrs
    J[b, a] = jrs
    jabs = float((L.abs().t() @ (L.abs() @ dw.abs())).max())
    K = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    kabs = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    for m in range(M):
        S = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        S[a, b] = L[m]
        S[b, a] = L[m]
        X = S @ C
        K += X @ X.t()
        Xa = S.abs() @ C.abs()
        kabs += Xa @ Xa.t()
    r = C.shape[1]
    return J, K, 2 * (L.shape[1] + M + r) * EPS * jabs, 2 * (2 * n + M * r) * EPS * float(kabs.max())


@pytest.mark.parametrize("natom,thrcom,ranks", [
    (2, 1e-6, (1, 7)),            # 28 functions: less than one tile
    (5, 1e-4, (8, 9, 63)),        # 70: a tile and a remainder
    (9, 1e-3, (64, 65)),          # 126
    (46, 0.3, (17, 129)),         # 644: many lower tiles, a remainder
])
def test_fp64_jk_at_tile_edges(natom, thrcom, ranks):
    g = MolGpu(B.make_molecule("edge", natom, [("3s2p1d", natom)], 3))
    g.cho_drv(thrcom=thrcom)
    Cs = [torch.from_numpy(B.density_factor(g.nbf, r, 40 + r)).cuda() for r in ranks]
    got = g.cho_jk_batch(Cs, precision=MolGpu.PREC_FP64)
    for C, (J, K) in zip(Cs, got):
        Jr, Kr, tj, tk = _reference(g, C)
        assert float((J - Jr).abs().max()) <= tj
        assert float((K - Kr).abs().max()) <= tk
        assert torch.equal(K, K.t()) and torch.equal(J, J.t())


def test_fp64_jk_column_tiles():
    """Ranks around the half-transform's column tiles (up to 64 columns, spread
    evenly, the last one cut to the eights of columns there are): every width of
    the last tile, and more columns than functions."""
    g = MolGpu(B.make_molecule("edge", 5, [("3s2p1d", 5)], 3))
    g.cho_drv(thrcom=1e-3)
    ranks = (56, 57, 64, 66, 80, 81, 111, 112, 113, 121, 168, 169, 177, 224, 225, 336)
    Cs = [torch.from_numpy(np.random.default_rng(r).standard_normal((g.nbf, r)) / np.sqrt(r)).cuda() for r in ranks]
    got = g.cho_jk_batch(Cs[:8], precision=MolGpu.PREC_FP64) + g.cho_jk_batch(Cs[8:], precision=MolGpu.PREC_FP64)
    for C, (J, K) in zip(Cs, got):
        Jr, Kr, tj, tk = _reference(g, C)
        assert float((J - Jr).abs().max()) <= tj
        assert float((K - Kr).abs().max()) <= tk
        assert torch.equal(K, K.t())
