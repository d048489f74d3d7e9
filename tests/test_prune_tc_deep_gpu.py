"""Deep protein trees whose likelihoods leave FP64's range, where the oracle's
unscaled FP64 gives no total: the tensor-core kernel's and the CUDA-core
kernel's per-pattern log likelihoods and their totals against pruning in FP64
that rescales every node (numpy).  Bounds as where FP64 needs no scaling: the total
within 1e-6 relative, patterns within 8 times the CUDA-core kernel's error, at
least 5e-5."""
import numpy
import pytest

from p4gpu import pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu
TENSOR_SHAPE, CORE_SHAPE = 3, 2


def _scaled(prob, codes, rates):
    """log likelihood per pattern; codes: raw character codes [taxon][pattern]."""
    t, sp = prob.tree, prob.parts[0]
    dim, nCat, nPat = sp.dim, sp.nCat, codes.shape[1]
    members = numpy.zeros((256, dim))   # states of code + 128
    for s in range(dim):
        members[s + 128, s] = 1.0
    members[[128 - 1, 128 - 2, 128 - 3]] = 1.0
    for k, row in enumerate(numpy.array(list(sp.equatesTable()), int).reshape(-1, dim)):
        members[128 - 64 + k] = row
    out = numpy.zeros((nCat, nPat))
    for c in range(nCat):
        cl, scale = {}, numpy.zeros(nPat)
        for v in t.postOrder:
            v = int(v)
            if v < 0:
                continue
            if t.isLeaf[v]:
                cl[v] = members[codes[t.seqNum[v]] + 128].T
                continue
            x = numpy.ones((dim, nPat))
            for k in t.children(v):
                k = int(k)
                P = sim.pmatrix(sp.rmats[sp.rMatrixNums[k]], sp.comps[sp.compNums[k]], t.brLen[k] * rates[c])
                x = x * (P @ cl.pop(k))
            m = x.max(0)
            scale += numpy.log(m)
            cl[v] = x / m
        out[c] = numpy.log(sp.comps[sp.compNums[t.root]] @ cl[t.root]) + scale
    top = out.max(0)
    return top + numpy.log(numpy.exp(out - top).sum(0) / nCat)


def _caterpillar(n):
    kids = {0: [1000, 1001, 1]}
    for k in range(1, n - 3):
        kids[k] = [2000 + k, k + 1]
    kids[n - 3] = [5000, 5001]
    return kids, 0


@pytest.mark.parametrize("taxa,sites,amb,mean", [(500, 140, 0.02, 0.1), (300, 30, 0.0, 0.8), (400, 129, 0.1, 0.4)])
def test_totals_of_deep_trees(taxa, sites, amb, mean, lib):
    rng = numpy.random.default_rng(taxa)
    kids, root = _caterpillar(taxa)
    t = sim.tree_from_children(kids, root, rng=rng, meanBrLen=mean)
    prob = sim.Problem(t, [sim.make_part(t, rng, "protein", sites, nComps=2, gammaShape=0.4, ambiguity=amb)], "deep")
    e = Engine(prob)
    e.setPrams()
    pf.setCladeSize(e.cTree, 0)
    nPat = e.nPatterns(0)
    pats, counts, _ = pf.getPatterns(e.cParts[0], prob.nTax, sites)
    want = _scaled(prob, numpy.asarray(pats)[:, :nPat].astype(int), pf.getGammaRates(e.cTree, 0, 0, 4))
    total = float((numpy.asarray(counts)[:nPat] * want).sum())
    assert want.min() < -745.0   # below the smallest FP64 number
    errs = {}
    for shape in (CORE_SHAPE, TENSOR_SHAPE):
        pf.setPruneShape(e.cTree, 0, shape)
        lnl = e.logLike(1)
        errs[shape] = numpy.abs(pf.getPatternLikes(e.cTree, 0, nPat)[2] - want).max()
        assert abs(lnl - total) <= 1e-6 * abs(total), shape
    assert errs[TENSOR_SHAPE] <= max(8.0 * errs[CORE_SHAPE], 5e-5)
    e.free()
