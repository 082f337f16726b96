"""The ERI launch rules and the branches of the bra half-transform: a class with
few work items (one CTA each, the largest tile), the same class with more items
than SMs (the throughput tiles), and tiles set by the caller must give the same
integrals.  The molecule has s to f shells with one to four contracted
functions, so odd and even numbers of bra products, classes with one or two
outputs per tile and shells of every bra range occur."""
import numpy as np
import pytest

from oracle import oracle as O
from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu, unique_quartets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mix", [[("4s3p2d1f_r", 1), ("2s1p", 1)], [("3s2p1d", 2)]])
def test_few_and_many_items_give_the_same_integrals(mix):
    mol = B.make_molecule("paths", 2, mix, 5)
    q = unique_quartets(len(mol.shells))
    g = MolGpu(mol)
    few, off = g.eri_quartets(q)
    few = few.cpu().numpy()
    n = 150  # every class has more items than the GPU has SMs
    many, moff = g.eri_quartets(np.tile(q, (n, 1)))
    many = many.cpu().numpy().reshape(n, -1)
    # the bar of the tile-choice tests: another order of the same sums
    tol = O.ERI_ABS_TOL * max(1.0, np.abs(few).max())
    assert np.array_equal(many, np.broadcast_to(many[0], many.shape))
    assert np.abs(many[0] - few).max() < tol
    g2 = MolGpu(mol, eri_tiles=None)
    for tpq, order in ((64, 0), (128, 1), (256, 3), (512, 2)):
        for a in range(7):
            for b in range(7):
                g2.set_eri_tile(a, b, tpq, order)
        got, _ = g2.eri_quartets(q)
        assert np.abs(got.cpu().numpy() - few).max() < tol
    o = O.Oracle(mol)
    rng = np.random.default_rng(1)
    for t in rng.choice(len(q), min(40, len(q)), replace=False):
        r = np.asarray(o.eri_quartet(*[int(v) for v in q[t]])).ravel(order="F")
        assert np.abs(few[off[t]:off[t + 1]] - r).max() < tol


def test_group_size_set_by_the_caller_holds():
    """A group size set by the caller is taken also where it leaves room for one
    primitive quartet a tile only (f f ket pairs: the planner's own groups give way
    to larger ones there), with the same integrals."""
    mol = B.make_molecule("held", 2, [("4s3p2d1f_r", 2)], 5)
    l = np.array([s.l for s in mol.shells])
    ff = [(i, j) for i in range(len(l)) for j in range(i + 1) if l[i] == l[j] == 3]
    pp = [(i, j) for i in range(len(l)) for j in range(i + 1) if l[i] == l[j] == 1]
    q = np.array([a + b for a in pp for b in ff], dtype=np.int32)
    g = MolGpu(mol)
    want = g.eri_quartets(q)[0]
    g.set_eri_tile(2, 6, 256, 0)
    g.eri_profile(True)
    got = g.eri_quartets(q)[0]
    tpq, pab, pcd = g.eri_class_times()[(2, 6)][1]
    assert tpq == 256 and pab * pcd < 4
    assert float((got - want).abs().max()) < O.ERI_ABS_TOL * max(1.0, float(want.abs().max()))
