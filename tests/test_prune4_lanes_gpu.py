"""The 4-state shapes that category counts have of their own: 14 and 15, two lanes
of two pairs for 6 categories, the middle pair formed by both; 13, for odd counts.
Everything per pattern has to be bitwise what shape 3 (one lane, which the
mirror test holds) gives: likelihoods, exponents, site rates, root partials
through the draws; with clade tables made by the shape and without.  Large trees
of 6 categories take the two lanes by themselves, smaller ones do not."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu

TILE = {13: 128, 14: 64, 15: 128}


def _outputs(e, n, nPat):
    e.setPrams()
    e.logLike(1)
    like, exps, lnl = pf.getPatternLikes(e.cTree, 0, nPat)
    rates, cats = pf.getSiteRates(e.cTree, e.cParts[0], 0, n)
    return [like.view(numpy.uint32), exps, lnl, rates, cats, pf.drawAncStates(e.cTree, 0, n, None, 3)]


@pytest.mark.parametrize("nCat,shape", [(6, 14), (6, 15), (3, 13), (5, 13)])
@pytest.mark.parametrize("taxa,sites,clades", [(9, 1, 0), (12, 65, 3), (40, 700, 4), (200, 129, 0)])
def test_bitwise(nCat, shape, taxa, sites, clades, lib):
    rng = numpy.random.default_rng(nCat * 1000 + taxa)
    t = sim.yule_tree(taxa, rng, meanBrLen=0.3)   # deep enough to rescale
    e = Engine(sim.Problem(t, [sim.make_part(t, rng, "dna", sites, nComps=2, nCat=nCat, ambiguity=0.1, pInvar=0.1)],
                           "lanes"))
    e.calcLogLike()
    pf.setCladeSize(e.cTree, clades)
    nPat = e.nPatterns(0)
    pf.setPruneShape(e.cTree, 0, 3)
    if clades:
        pf.setCladeShape(e.cTree, 0, 3)
    want = _outputs(e, sites, nPat)
    pf.setPruneShape(e.cTree, 0, shape)
    if clades:
        pf.setCladeShape(e.cTree, 0, shape)
    assert pf.getPruneShape(e.cTree, 0) == (shape, TILE[shape])
    for a, b in zip(want, _outputs(e, sites, nPat)):
        assert numpy.array_equal(numpy.asarray(a), numpy.asarray(b))
    e.free()


@pytest.mark.parametrize("taxa", [420, 470, 900])
def test_large_trees_of_six_categories(taxa, lib):
    rng = numpy.random.default_rng(taxa)
    t = sim.yule_tree(taxa, rng, meanBrLen=0.02)
    e = Engine(sim.Problem(t, [sim.make_part(t, rng, "dna", 80, nCat=6)], "lanes"))
    lnl = e.calcLogLike()
    pf.setCladeSize(e.cTree, 0)   # nothing fits but what reads its decks through L1
    assert abs(e.calcLogLike() - lnl) <= 1e-12 * abs(lnl)
    if taxa == 900:
        assert pf.getPruneShape(e.cTree, 0)[0] in (14, 15)
    pf.setPrecision(e.cTree, 1)
    assert abs(e.calcLogLike() - lnl) <= 1e-6 * abs(lnl)
    e.free()


def test_other_counts_have_no_shared_pair(lib):
    rng = numpy.random.default_rng(2)
    t = sim.yule_tree(9, rng)
    for nCat in (1, 2, 3, 4, 5, 8):
        e = Engine(sim.Problem(t, [sim.make_part(t, rng, "dna", 50, nCat=nCat)], "lanes"))
        e.calcLogLike()
        for shape in (14, 15, 16):
            with pytest.raises(P4Error):
                pf.setPruneShape(e.cTree, 0, shape)
        e.free()
