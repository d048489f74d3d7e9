"""P(t) = e^(Qt) of a normalised reversible rate matrix to some 40 digits, for
models so skewed that an FP64 eigensystem is no reference: scaling, Taylor's
series and squaring in decimal arithmetic."""
import decimal

import numpy

DIGITS = 60


def _matmul(a, b):
    cols = list(zip(*b))
    return [[sum(x * y for x, y in zip(row, col)) for col in cols] for row in a]


def rate_matrix(R, pi):
    """R.diag(pi), rows summing to zero, mean rate one, from the exact values of
    the doubles given (R's diagonal is not read)."""
    n = len(pi)
    D = decimal.Decimal
    with decimal.localcontext() as c:
        c.prec = DIGITS
        p = [D(float(x)) for x in pi]
        q = [[D(float(R[i][j])) * p[j] if i != j else D(0) for j in range(n)] for i in range(n)]
        for i in range(n):
            q[i][i] = -sum(q[i])
        mean = -sum(p[i] * q[i][i] for i in range(n))
        return [[x / mean for x in row] for row in q]


def pmatrix(Q, t):
    """e^(Qt), Q from rate_matrix, rounded to FP64."""
    n = len(Q)
    D = decimal.Decimal
    with decimal.localcontext() as c:
        c.prec = DIGITS
        a = [[x * D(float(t)) for x in row] for row in Q]
        norm = max(sum(abs(x) for x in row) for row in a)
        k = 0
        while norm > D("0.001"):
            norm /= 2
            k += 1
        a = [[x / (1 << k) for x in row] for row in a]
        term = [[D(int(i == j)) for j in range(n)] for i in range(n)]
        out = [row[:] for row in term]
        for m in range(1, 40):
            term = [[x / m for x in row] for row in _matmul(term, a)]
            out = [[x + y for x, y in zip(u, v)] for u, v in zip(out, term)]
            if max(abs(x) for row in term for x in row) < D(10) ** -(DIGITS - 5):
                break
        for _ in range(k):
            out = _matmul(out, out)
        return numpy.array([[float(x) for x in row] for row in out])
