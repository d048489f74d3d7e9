"""The FP64 path where its blocks' chunks end: every number of categories that
gives a chunk of its own, pattern counts below, at and above a multiple of it.
Oracle: the CPU restatement of the reference's FP64 pruning, on its own P.
Tolerance: 1e-10 of the lnL (P decks to 1e-12 of each other, as the fixtures',
through the ten branches of a site's product)."""
import numpy
import pytest

from p4gpu import pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nCat", [1, 2, 3, 4, 5, 7, 8, 12, 16])
@pytest.mark.parametrize("data,sites", [("dna", 1), ("dna", 300), ("dna", 1030), ("protein", 3), ("protein", 260)])
def test_against_the_oracle(data, sites, nCat, lib, port):
    rng = numpy.random.default_rng(nCat + sites)
    t = sim.yule_tree(6, rng, 0.8)
    prob = sim.Problem(t, [sim.make_part(t, rng, data, sites, nCat=nCat, pInvar=0.1, ambiguity=0.02)], "chunks")
    e = Engine(prob)
    pf.setPrecision(e.cTree, 1)
    want, _ = port.port_loglike64(prob)
    got = e.calcLogLike()
    assert abs(got - want) <= 1e-10 * abs(want)
    assert e.calcLogLike() == got
    e.free()
