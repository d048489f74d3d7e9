"""A program that outgrows the tile shape in use (clade tables turned off, a
topology with fewer clades): the smaller shape that then runs has tiles of its
own, so the lnL is that of the FP64 path, for setPrams and without it."""
import numpy
import pytest

from p4gpu import P4Error, pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


def _engine(data, taxa, sites, nCat, seed):
    rng = numpy.random.default_rng(seed)
    t = sim.yule_tree(taxa, rng, meanBrLen=0.02)
    sp = sim.make_part(t, rng, data, 4, nCat=nCat)
    base = rng.integers(4, size=sites)
    sp.sequences = ["".join(sp.symbols[s] for s in numpy.where(rng.random(sites) < 0.05, rng.integers(4, size=sites), base))
                    for _ in range(taxa)]
    return Engine(sim.Problem(t, [sp], "retile"))


def _lnl64(e):
    pf.setPrecision(e.cTree, 1)
    v = e.calcLogLike()
    pf.setPrecision(e.cTree, 0)
    return v


@pytest.mark.parametrize("taxa,nCat", [(390, 6), (450, 4), (400, 3), (650, 2)])
@pytest.mark.parametrize("setPrams", [True, False])
def test_clade_tables_off(taxa, nCat, setPrams, lib):
    e = _engine("dna", taxa, 700, nCat, taxa + nCat)
    want = _lnl64(e)
    retiled = 0
    for size in (8, 4):
        for shape in range(13):
            pf.setCladeSize(e.cTree, size)
            e.calcLogLike()
            try:
                pf.setPruneShape(e.cTree, 0, shape)
            except P4Error:
                continue
            tile = pf.getPruneShape(e.cTree, 0)[1]
            assert abs(e.calcLogLike() - want) <= 1e-6 * abs(want), (size, shape)
            pf.setCladeSize(e.cTree, 0)
            got = e.calcLogLike() if setPrams else e.logLike(0)
            assert abs(got - want) <= 1e-6 * abs(want), (size, shape)
            retiled += pf.getPruneShape(e.cTree, 0)[1] != tile
    assert retiled > 0
    e.free()


def test_clade_tables_off_protein(lib):
    e = _engine("protein", 300, 700, 4, 7)
    want = _lnl64(e)
    for size in (6, 0, 4, 0):
        pf.setCladeSize(e.cTree, size)
        assert abs(e.calcLogLike() - want) <= 1e-6 * abs(want), size
    e.free()


def test_topology_with_fewer_clades(lib):
    """A caterpillar on the same nodes: its only clade is at the tip."""
    e = _engine("dna", 450, 700, 4, 454)
    first = e.calcLogLike()
    t = e.problem.tree
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
    assert not take
    e.setTopologyArrays(parent, left, sib, t.root)
    want = _lnl64(e)
    retiled = 0
    for size, shape in [(a, b) for a in (8, 4) for b in range(13)]:
        pf.setCladeSize(e.cTree, size)
        e.setTopologyArrays(t.parent, t.leftChild, t.sibling, t.root)
        assert abs(e.calcLogLike() - first) <= 1e-9 * abs(first)
        try:
            pf.setPruneShape(e.cTree, 0, shape)
        except P4Error:
            continue
        tile = pf.getPruneShape(e.cTree, 0)[1]
        e.setTopologyArrays(parent, left, sib, t.root)
        assert abs(e.calcLogLike() - want) <= 1e-6 * abs(want), shape
        retiled += pf.getPruneShape(e.cTree, 0)[1] != tile
    assert retiled > 0
    e.free()
