"""treeInfo between a new topology and an evaluation without setPrams leaves the
evaluation what it is without it."""
import numpy
import pytest

from p4gpu import pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("data", ["dna", "protein"])
def test_tree_info_after_a_new_topology(data, lib):
    rng = numpy.random.default_rng(2)
    t = sim.yule_tree(12, rng)
    prob = sim.Problem(t, [sim.make_part(t, rng, data, 200)], "info")
    first = Engine(prob)
    other = Engine(prob, shared=(first.cData, first.cParts))
    inner = [v for v in range(t.nNodes) if not t.isLeaf[v] and v != t.root and t.parent[v] != t.root]
    v = inner[0]
    aunt = next(c for c in t.children(t.parent[v]) if c != v)
    t2 = t.swapped(next(iter(t.children(v))), aunt)
    for e in (first, other):
        for _ in range(2):
            old = e.calcLogLike()
        e.setTopologyArrays(t2.parent, t2.leftChild, t2.sibling, t2.root)
    pf.treeInfo(other.cTree)
    want = first.logLike(0)
    assert want != old
    assert other.logLike(0) == want
    other.free()
    first.free()
