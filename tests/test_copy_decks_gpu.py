"""p4_copyBigPDecks: a tree evaluated on another tree's P decks gives that
tree's lnL (same model and topology; the branch lengths, which only the decks
hold, differ).  The pruning kernels read the decks in two forms, the FP32
decks and the tensor-core kernel's images of them.  Tolerance: 1e-6 of the
lnL, the FP32 pruning's; the trees' own lnLs are far further apart."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


def _pair(data):
    rng = numpy.random.default_rng(3)
    t = sim.yule_tree(11, rng)
    prob = sim.Problem(t, [sim.make_part(t, rng, data, 150)], "copy")
    a = Engine(prob)
    b = Engine(prob, shared=(a.cData, a.cParts))
    a.setBrLens(t.brLen * 3.0)
    return a, b


@pytest.mark.parametrize("data,shape", [("dna", 0), ("protein", 0), ("protein", 3)])
def test_the_copy_takes_every_form_of_the_decks(data, shape, lib):
    a, b = _pair(data)
    want, own = a.calcLogLike(), b.calcLogLike()
    assert abs(want - own) > 1e-3 * abs(own)
    for e in (a, b):
        pf.setPruneShape(e.cTree, 0, shape)
    pf.p4_copyBigPDecks(a.cTree, b.cTree, 1)
    assert abs(b.logLike() - want) <= 1e-6 * abs(want)
    assert abs(b.calcLogLike() - own) <= 1e-6 * abs(own)    # and its own again with its own setPrams
    b.free()
    a.free()


@pytest.mark.parametrize("data", ["dna", "protein"])
def test_into_a_tree_that_never_set_its_parameters(data, lib):
    a, b = _pair(data)
    want = a.calcLogLike()
    pf.p4_copyBigPDecks(a.cTree, b.cTree, 1)
    assert abs(b.logLike() - want) <= 1e-6 * abs(want)
    b.free()
    a.free()


def test_from_a_tree_without_parameters_is_refused(lib):
    a, b = _pair("dna")
    with pytest.raises(P4Error):
        pf.p4_copyBigPDecks(a.cTree, b.cTree, 1)
    with pytest.raises(P4Error):
        b.logLike()
    b.free()
    a.free()
