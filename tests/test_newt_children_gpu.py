"""Newton branch lengths on trees whose nodes have as many children as a
round's records hold: 17, since a branch has at most 16 siblings; 18 are
refused.  Oracle: the FP64 evaluation of the same library.  A round ends when
lnL moves by less than likeDelta, and no single branch is then worth more than
20 times that (the branches moved after it included), so moving one by 2 %
gains at most 20 likeDelta, plus the rounding of two lnLs."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu

DELTA = 1e-7


def _engine(rootKids, innerKids):
    rng = numpy.random.default_rng(rootKids + 100 * innerKids)
    first = rootKids + 1
    t = sim.tree_from_children({0: list(range(1, first)), 2: list(range(first, first + innerKids))}, 0, rng=rng,
                               meanBrLen=0.2)
    e = Engine(sim.Problem(t, [sim.make_part(t, rng, "dna", 200)], "children"))
    pf.setPrecision(e.cTree, 1)
    return e, t


@pytest.mark.parametrize("rootKids,innerKids", [(3, 16), (3, 17), (17, 2), (17, 17)])
def test_as_many_children_as_fit(rootKids, innerKids, lib):
    e, t = _engine(rootKids, innerKids)
    start = e.calcLogLike()
    pf.p4_newtAround(e.cTree, 1e-5, DELTA)
    bl = pf.p4_getBrLens(e.cTree, t.nNodes)
    best = e.calcLogLike()
    assert best > start
    for v in range(t.nNodes):
        if v == t.root or not 1e-5 < bl[v] < 2.9:
            continue
        for f in (0.98, 1.02):
            b = bl.copy()
            b[v] *= f
            e.setBrLens(b)
            assert e.calcLogLike() <= best + 20 * DELTA + 2e-15 * abs(best), (v, f)
    e.free()


@pytest.mark.parametrize("rootKids,innerKids", [(3, 18), (18, 2)])
def test_one_more_is_refused(rootKids, innerKids, lib):
    e, t = _engine(rootKids, innerKids)
    with pytest.raises(P4Error, match="16 siblings"):
        pf.p4_newtAround(e.cTree, 1e-5, DELTA)
    e.free()
