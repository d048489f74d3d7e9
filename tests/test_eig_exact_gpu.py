"""P decks of skewed and close-spectrum models against e^(Qt) to 40 digits
(tests/exact_expm.py), for which an FP64 eigensystem is itself no reference.

Tolerance, from the method: P = diag(1/sq) X e X^T diag(sq), so an error of X's
and lambda's goes into P_ij times sqrt(pi_j / pi_i).  The refinement is accepted
with each unresolved pair coupled by up to 256 eps ||A||, which moves e^(At) by
that times t, for at most n pairs with one state; the pair arithmetic of the decks
adds 64 eps (2^-46).  So |dP_ij| <= 256 n eps (1 + ||A|| t) sqrt(pi_j / pi_i)."""
import numpy
import pytest

import exact_expm
from p4gpu import pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


def model(dim, kind, rng):
    k = dim * (dim - 1) // 2
    pi, u = rng.dirichlet(numpy.full(dim, 5.0)), rng.dirichlet(numpy.full(k, 2.0)) + 1e-6
    if kind == "skewed":
        pi, u = rng.dirichlet(numpy.full(dim, 0.3)) + 1e-5, numpy.exp(rng.normal(0, 2, k))
    if kind == "rare":        # one state at p4's smallest composition value
        pi[rng.integers(dim)] = 1e-13
    if kind == "flat":
        pi, u = numpy.full(dim, 1.0 / dim), 1.0 + 0.5 * rng.random(k)
    if kind == "near":
        pi, u = numpy.full(dim, 1.0 / dim), 1.0 + rng.choice([1e-4, 1e-6, 1e-9, 1e-13]) * rng.random(k)
    return sim._fix(pi / pi.sum()), sim.sym_from_upper(u / u.sum(), dim)


def tolerance(Q, pi, t):
    sq = numpy.sqrt(pi)
    A = sq[:, None] * numpy.array([[float(x) for x in row] for row in Q]) / sq[None, :]
    return 256 * len(pi) * numpy.finfo(float).eps * (1 + numpy.linalg.norm(A) * t) * sq[None, :] / sq[:, None]


@pytest.mark.parametrize("kind", ["random", "skewed", "rare", "flat", "near"])
@pytest.mark.parametrize("dim", [4, 20])
def test_decks(dim, kind, lib):
    rng = numpy.random.default_rng([dim, len(kind)])
    t = sim.yule_tree(4, rng)
    for _ in range(12 if dim == 4 else 3):
        pi, R = model(dim, kind, rng)
        sp = sim.make_part(t, rng, "dna" if dim == 4 else "protein", 32, nCat=1)
        sp.comps, sp.rmats = pi[None, :], R[None]
        e = Engine(sim.Problem(t, [sp], kind))
        e.calcLogLike()
        Q = exact_expm.rate_matrix(R, pi)
        for v in range(1, 4 if dim == 4 else 2):
            bl = t.brLen[v]
            err = numpy.abs(pf.getPDeck(e.cNodes[v], 0, 0, dim) - exact_expm.pmatrix(Q, bl))
            assert (err <= tolerance(Q, pi, bl)).all(), (err / tolerance(Q, pi, bl)).max()
        e.free()
