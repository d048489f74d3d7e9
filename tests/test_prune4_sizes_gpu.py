"""The largest 4-state trees a category count can be evaluated on, and the
sizes to which each tile shape can be pinned: both are bounded by the shared
memory a tile needs, whose first forms (codes of the tile's patterns, stack
slots, P decks of 16 floats a category where they are staged) set the limits.
Oracle: the FP64 path on the same tree, to 1e-6 of the lnL (the FP32
pruning's tolerance); the shapes among themselves to 1e-12 (the same
per-pattern values, added in another order)."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu

SITES = 40


def _engine(kind, n, nCat):
    rng = numpy.random.default_rng(n + nCat)
    if kind == "yule":
        t = sim.yule_tree(n, rng, 0.02)
    else:   # a caterpillar
        kids = {v: [100000 + v, v + 1] for v in range(n - 3)}
        kids[n - 3] = [200000, 200001, 200002]
        t = sim.tree_from_children(kids, 0, rng=rng, meanBrLen=0.02)
    sp = sim.make_part(t, rng, "dna", 4, nCat=nCat)
    base = rng.integers(4, size=SITES)
    sp.sequences = []
    for _ in range(n):
        x = numpy.where(rng.random(SITES) < 0.02, rng.integers(4, size=SITES), base)
        sp.sequences.append("".join("acgt"[s] for s in x))
    return Engine(sim.Problem(t, [sp], "sizes"))


@pytest.mark.parametrize("nCat,kind,n", [(1, "yule", 800), (1, "cat", 790), (2, "yule", 1500), (2, "cat", 1800),
                                         (3, "yule", 700), (4, "cat", 1800), (5, "yule", 600), (6, "yule", 1200),
                                         (6, "cat", 1500), (8, "yule", 1500)])
def test_large_trees_are_evaluated(nCat, kind, n, lib):
    e = _engine(kind, n, nCat)
    lnl = e.calcLogLike()
    assert e.calcLogLike() == lnl
    pf.setPrecision(e.cTree, 1)
    assert abs(lnl - e.calcLogLike()) <= 1e-6 * abs(lnl)
    e.free()


# (threads, tile, decks staged, category counts) of each shape's first form
FIRST = [(128, 128, 1, 1), (128, 256, 1, 1), (256, 256, 1, 1), (256, 256, 0, 1), (128, 256, 0, 1), (512, 512, 0, 1),
         (256, 64, 0, 4), (256, 128, 0, 2), (128, 64, 0, 2), (256, 64, 1, 4), (512, 128, 0, 4), (256, 256, 1, 34),
         (128, 256, 1, 34)]


@pytest.mark.parametrize("nCat,kind,n", [(1, "cat", 500), (1, "yule", 750), (2, "cat", 1200), (3, "cat", 300),
                                         (3, "yule", 500), (4, "cat", 300), (4, "yule", 700), (4, "cat", 1500),
                                         (6, "yule", 700), (8, "yule", 300), (8, "cat", 500)])
def test_shapes_can_be_pinned_where_they_could(nCat, kind, n, lib):
    e = _engine(kind, n, nCat)
    pf.setCladeSize(e.cTree, 0)
    lnl = e.calcLogLike()
    info = pf.treeInfo(e.cTree)
    for shape, (threads, tile, staged, counts) in enumerate(FIRST):
        need = info["nProg"] * 16 + staged * (e.problem.tree.nNodes - 1) * nCat * 64 + (n * tile + 15) // 16 * 16 \
            + 16 + info["nSlots"] * nCat * 16 * tile + threads // 32 * 8 + 16
        if (nCat in (3, 4) if counts == 34 else nCat % counts == 0) and need <= 227 * 1024:
            pf.setPruneShape(e.cTree, 0, shape)
            assert abs(e.calcLogLike() - lnl) <= 1e-12 * abs(lnl), shape
        else:
            with pytest.raises(P4Error):
                pf.setPruneShape(e.cTree, 0, shape)
    e.free()


@pytest.mark.parametrize("nCat,n", [(1, 600), (3, 320), (5, 210)])
def test_odd_counts_take_no_more_than_their_categories(nCat, n, lib):
    """A staged shape that fits with 16 floats a category (and a row of ones) runs
    itself, not a smaller one in its place."""
    e = _engine("yule", n, nCat)
    pf.setCladeSize(e.cTree, 0)
    lnl = e.calcLogLike()
    info = pf.treeInfo(e.cTree)
    for shape in (0, 1, 2):
        threads, tile, _, _ = FIRST[shape]
        need = info["nProg"] * 16 + (e.problem.tree.nNodes + 1) * nCat * 64 + (n * tile + 15) // 16 * 16 + 16 \
            + info["nSlots"] * nCat * 16 * tile + threads // 32 * 8 + 16
        assert shape != 0 or need <= 227 * 1024
        if need <= 227 * 1024:
            pf.setPruneShape(e.cTree, 0, shape)
            assert pf.getPruneShape(e.cTree, 0) == (shape, tile)
            assert abs(e.calcLogLike() - lnl) <= 1e-12 * abs(lnl), shape
    e.free()


@pytest.mark.parametrize("nCat", [1, 3, 5])
def test_the_smallest_shape_of_odd_counts(nCat, lib):
    e = _engine("yule", 60, nCat)
    lnl = e.calcLogLike()
    pf.setPruneShape(e.cTree, 0, 13)
    assert pf.getPruneShape(e.cTree, 0) == (13, 128)
    assert abs(e.calcLogLike() - lnl) <= 1e-12 * abs(lnl)
    e.free()


@pytest.mark.parametrize("nCat", [2, 3, 4])
def test_clade_shapes_can_be_pinned_on_large_trees(nCat, lib):
    e = _engine("yule", 600, nCat)
    lnl = e.calcLogLike()
    pf.setCladeSize(e.cTree, 4)
    for shape in range(13):
        try:
            pf.setCladeShape(e.cTree, 0, shape)
        except P4Error:
            continue
        if shape in (0, 1, 2, 9, 11, 12):   # these staged every deck from the first
            continue
        assert abs(e.calcLogLike() - lnl) <= 1e-12 * abs(lnl), shape
    e.free()
