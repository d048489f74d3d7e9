"""A batch that refuses a tree whose new topology outgrows its tile shape leaves
that tree's tiles as they are: the tree evaluates alone, and the batch takes it
again once its topology fits."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


def _caterpillar(t):
    """(parent, leftChild, sibling) of a caterpillar on t's nodes."""
    parent, left, sib = (numpy.full(t.nNodes, -1, numpy.int32) for _ in range(3))
    chain = [t.root] + [v for v in range(t.nNodes) if not t.isLeaf[v] and v != t.root]
    take = [v for v in range(t.nNodes) if t.isLeaf[v]]
    for k, v in enumerate(chain):
        ch = [take.pop()] if k else [take.pop(), take.pop()]
        ch.append(chain[k + 1] if k + 1 < len(chain) else take.pop())
        left[v] = ch[0]
        for a, b in zip(ch[:-1], ch[1:]):
            sib[a] = b
        for c in ch:
            parent[c] = v
    return parent, left, sib


def test_refused_tree_keeps_its_tiles(lib):
    rng = numpy.random.default_rng(6)
    t = sim.yule_tree(200, rng, meanBrLen=0.02)
    sp = sim.make_part(t, rng, "dna", 1500)
    prob = sim.Problem(t, [sp], "batch")
    pf.setAutotune(False)
    try:
        es = [Engine(prob)]
        es.append(Engine(prob, shared=(es[0].cData, es[0].cParts)))
        cat = _caterpillar(t)
        for e in es:
            pf.setCladeSize(e.cTree, 0)
            e.setTopologyArrays(*cat, t.root)
        want = es[0].calcLogLike()
        pf.setPruneShape(es[0].cTree, 0, 5)   # 512 patterns: a stack slot of 4 categories is 32 KB
        assert pf.getPruneShape(es[0].cTree, 0) == (5, 512)
        batch = pf.Batch([e.cTree for e in es])
        numpy.testing.assert_allclose(batch.logLike(), [want, want], rtol=1e-12)
        es[1].setTopologyArrays(t.parent, t.leftChild, t.sibling, t.root)   # needs more stack slots
        with pytest.raises(P4Error, match="does not fit"):
            batch.logLike()
        yule = es[1].calcLogLike()
        pf.setPrecision(es[1].cTree, 1)
        assert abs(es[1].calcLogLike() - yule) <= 1e-6 * abs(yule)
        pf.setPrecision(es[1].cTree, 0)
        es[1].setTopologyArrays(*cat, t.root)
        for _ in range(2):
            numpy.testing.assert_allclose(batch.logLike(), [want, want], rtol=1e-12)
        batch.free()
    finally:
        pf.setAutotune(True)
    for e in reversed(es):
        e.free()
