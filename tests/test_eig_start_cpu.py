"""The FP32 Jacobi start of the setPrams eigensystems (csrc/p4g_pmat.cu) replayed
in numpy's FP32, with its orders and its stopping rules, followed by the FP64
refinement and its acceptance rule (test_pair_numerics_cpu.py), against e^(Qt)
to 40 digits:

  - more than 4 states: sweeps in round-robin order until every |s_ij| is at most
    3e-6 of its eigenvalues' gap or 1e-8 ||A||, twelve at most;
  - 4 states (eig4Warp): six rotations a sweep in a fixed order until the
    off-diagonal mass is 1e-13 of the diagonal's, twelve at most.

What the rule accepts has to be within test_eig_exact_gpu.py's tolerance; models
without close eigenvalues have to be accepted, so that they never need the FP64
sweeps.  The kernel's reciprocal square root is good to 2^-22 instead of 2^-24:
replayed here by dropping two bits."""
import numpy
import pytest

import exact_expm
from test_eig_exact_gpu import model, tolerance
from test_pair_numerics_cpu import refine, symmetric_form

f32 = numpy.float32


def rsqrt(x):
    y = f32(1.0) / numpy.sqrt(f32(x))
    return (numpy.array(y, f32).view(numpy.uint32) & numpy.uint32(0xfffffffc)).view(f32)[()]


def rotation(app, aqq, apq):
    dd, r2 = f32(aqq - app), f32(2) * apq
    h = f32(dd * dd + r2 * r2)
    if r2 == 0 or h < f32(1e-36):
        return f32(1), f32(0)
    u = f32(abs(dd) + h * rsqrt(h))
    inv = rsqrt(f32(u * u + r2 * r2))
    return f32(u * inv), f32((r2 if dd >= 0 else -r2) * inv)


def apply_pairs(S, U, pairs):
    """One round: the rotations of disjoint pairs, found before any is applied."""
    J = numpy.eye(len(S), dtype=f32)
    for p, q in pairs:
        c, s = rotation(S[p, p], S[q, q], S[p, q])
        J[p, p] = J[q, q] = c
        J[p, q], J[q, p] = s, -s
    S = (J.T @ (S @ J)).astype(f32)
    return (numpy.triu(S) + numpy.triu(S, 1).T).astype(f32), (U @ J).astype(f32)


def start_large(A):
    n = len(A)
    m = n + n % 2
    S, U = A.astype(f32), numpy.eye(n, dtype=f32)
    tiny = f32(1e-8) * f32(numpy.linalg.norm(S))
    for _ in range(12):
        gap = numpy.abs(numpy.diag(S)[:, None] - numpy.diag(S)[None, :])
        v = numpy.abs(S)
        if not (numpy.triu(~((v <= tiny) | (v <= f32(3e-6) * gap)), 1)).any():
            break
        order = list(range(m))
        for _ in range(m - 1):
            pairs = [(order[i], order[m - 1 - i]) for i in range(m // 2)]
            S, U = apply_pairs(S, U, [(min(x), max(x)) for x in pairs if max(x) < n])
            order = [order[0], order[-1]] + order[1:-1]
    return U


def start_four(A):
    S, U = A.astype(f32), numpy.eye(4, dtype=f32)
    for _ in range(12):
        dg, off = (numpy.diag(S) ** 2).sum(), (numpy.triu(S, 1) ** 2).sum()
        if off <= f32(1e-13) * dg or off == 0:
            break
        for p, q in ((0, 3), (1, 2), (0, 2), (1, 3), (0, 1), (2, 3)):
            S, U = apply_pairs(S, U, [(p, q)])
    return U


@pytest.mark.parametrize("kind", ["random", "skewed", "rare", "flat", "near"])
@pytest.mark.parametrize("dim", [4, 20])
def test_start_and_refinement(dim, kind):
    rng = numpy.random.default_rng([dim, len(kind), 1])
    accepted = 0
    tries = 40 if dim == 4 else 3
    for _ in range(tries):
        pi, R = model(dim, kind, rng)
        A, sq = symmetric_form(R, pi)
        U = start_four(A) if dim == 4 else start_large(A)
        X, lam, ok = refine(A, U.astype(float), numpy.linalg.norm(A))
        if not ok:
            continue
        accepted += 1
        Q = exact_expm.rate_matrix(R, pi)
        for t in ((0.02, 0.7) if dim == 4 else (0.2,)):
            P = (X * numpy.exp(lam * t)) @ X.T * sq[None, :] / sq[:, None]
            err = numpy.abs(P - exact_expm.pmatrix(Q, t))
            assert (err <= tolerance(Q, pi, t)).all(), (err / tolerance(Q, pi, t)).max()
    if kind == "random":
        assert accepted == tries
