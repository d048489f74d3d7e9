"""The buffers an ancestral draw keeps between calls belong to the data: any
number of trees on one alignment share them.  24 trees of 400,000 sites in a few patterns
would hold 77 MB of uniforms on the device if each kept its own (a tree's
other buffers follow its few patterns); one set is 3.2 MB, counted here with
a margin of 16 MB for the trees."""
import numpy
import pytest

from p4gpu import pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


def _engines(n, sites):
    rng = numpy.random.default_rng(8)
    t = sim.yule_tree(5, rng)
    sp = sim.make_part(t, rng, "dna", 50)
    sp.sequences = [s * (sites // 50) for s in sp.sequences]
    prob = sim.Problem(t, [sp], "draws")
    first = Engine(prob)
    return [first] + [Engine(prob, shared=(first.cData, first.cParts)) for _ in range(n - 1)]


def test_trees_share_the_buffers(lib):
    import torch
    sites = 400000
    es = _engines(24, sites)
    u = numpy.random.default_rng(1).random(sites)
    for e in es:
        e.calcLogLike()
    want = pf.drawAncStates(es[0].cTree, 0, sites, u)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for e in es[1:]:
        assert numpy.array_equal(pf.drawAncStates(e.cTree, 0, sites, u), want)
    assert free0 - torch.cuda.mem_get_info()[0] < 16 << 20
    for e in reversed(es):
        e.free()
