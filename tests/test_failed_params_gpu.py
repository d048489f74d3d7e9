"""Model values whose rates or eigensystem cannot be formed are refused at
every evaluation, not at the first alone, and leave nothing behind: the tree
then evaluates good values as one that never saw the others.  An R matrix of
zeros has no normalised Q; the incomplete gamma's series for a shape of 1e12
is cut off after 200,000 terms."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


def _engine(data="dna", shared=None, seed=5):
    rng = numpy.random.default_rng(seed)
    t = sim.yule_tree(6, rng)
    return Engine(sim.Problem(t, [sim.make_part(t, rng, data, 40)], "failed"), shared=shared)


def _spoil(e, what):
    if what == "shape":
        e.setGamma(0, 0, 1e12)
    else:
        sp = e.problem.parts[0]
        e.setRMatrix(0, 0, numpy.zeros(sp.dim * (sp.dim - 1) // 2))


def _repair(e):
    sp = e.problem.parts[0]
    e.setGamma(0, 0, sp.gammaShapes[0])
    e.setRMatrix(0, 0, sim.upper_of(sp.rmats[0]))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("data,what", [("dna", "shape"), ("dna", "matrix"), ("protein", "matrix")])
def test_refused_every_time(data, what, precision, lib):
    e = _engine(data)
    pf.setPrecision(e.cTree, precision)
    good = e.calcLogLike()
    _spoil(e, what)
    for _ in range(3):
        with pytest.raises(P4Error, match="did not converge"):
            e.calcLogLike()
    _repair(e)
    assert e.calcLogLike() == good
    e.free()


@pytest.mark.parametrize("what", ["shape", "matrix"])
def test_failed_evaluation_keeps_the_site_likelihoods(what, lib):
    e = _engine()
    e.setPrams()
    e.logLike(1)
    want = pf.getSiteLikes(e.cParts[0], 40)
    _spoil(e, what)
    for _ in range(2):
        e.setPrams()
        with pytest.raises(P4Error, match="did not converge"):
            e.logLike(1)
        assert numpy.array_equal(pf.getSiteLikes(e.cParts[0], 40), want)
    _repair(e)
    e.setBrLens(e.problem.tree.brLen * 1.5)
    e.setPrams()
    e.logLike(1)
    assert (pf.getSiteLikes(e.cParts[0], 40) != want).any()
    e.free()


def test_every_failure_of_a_batch_call_is_taken(lib):
    a = _engine()
    b = _engine(shared=(a.cData, a.cParts))
    good = [e.calcLogLike() for e in (a, b)]
    for e in (a, b):
        _spoil(e, "matrix")
    with pytest.raises(P4Error, match="did not converge"):
        pf.treeLogLikeBatch([a.cTree, b.cTree])
    for e in (a, b):
        _repair(e)
    assert [e.calcLogLike() for e in (a, b)] == good
    b.free()
    a.free()
