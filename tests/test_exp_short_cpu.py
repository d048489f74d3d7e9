"""expShort (csrc/p4g_math.cuh), the exponential of the Newton steps and the
gamma rates, against e^x to 40 digits: within 1.5 ulp from -708 up to 700, where
it hands over to exp(), 0 below.  The same source for the host; its operations
(IEEE products, sums and FMAs) are the device's, and neither compiler may
contract what is left, since no bare product feeds a sum."""
import ctypes
import decimal
import math
import os
import subprocess

import numpy
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exp_short(tmp_path_factory):
    d = tmp_path_factory.mktemp("exp_short")
    src, so = str(d / "e.cpp"), str(d / "e.so")
    with open(src, "w") as f:
        f.write('#include "p4g_math.cuh"\n'
                'extern "C" void run(const double *x, double *y, int n)\n'
                '{ for (int i = 0; i < n; i++) y[i] = p4g::expShort(x[i]); }\n')
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(REPO, "p4-phylogenetics_gb300", "csrc"), src, "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def run(x):
        x = numpy.ascontiguousarray(x, numpy.double)
        y = numpy.empty_like(x)
        p = ctypes.POINTER(ctypes.c_double)
        lib.run(x.ctypes.data_as(p), y.ctypes.data_as(p), len(x))
        return y
    return run


def _points():
    rng = numpy.random.default_rng(3)
    edges = []   # where k changes, and the range's ends, a few ulps to either side
    for k in range(-1021, 1010, 7):
        edges.append((k + 0.5) * math.log(2.0))
    edges += [-708.0, 700.0, 0.0, -1e-300, 1e-300]
    edges = numpy.array(edges)
    near = [edges]
    for way in (-numpy.inf, numpy.inf):
        e = edges
        for _ in range(3):
            e = numpy.nextafter(e, way)
            near.append(e)
    x = numpy.concatenate(near + [rng.uniform(-708.0, 700.0, 4000), -numpy.exp(rng.uniform(-30.0, 6.5, 4000))])
    return x[(x >= -708.0) & (x < 700.0)]


def test_ulps(exp_short):
    x = _points()
    worst = decimal.Decimal(0)
    with decimal.localcontext() as c:
        c.prec = 40
        for a, y in zip(x, exp_short(x)):
            want = decimal.Decimal(float(a)).exp()
            worst = max(worst, abs(decimal.Decimal(float(y)) - want) / decimal.Decimal(math.ulp(float(want))))
    assert worst <= 1.5, worst


def test_outside(exp_short):
    below = [numpy.nextafter(-708.0, -numpy.inf), -709.0, -1e4, -1e308, -numpy.inf]
    assert (exp_short(below) == 0.0).all()
    y = exp_short([700.0, 710.0, numpy.inf, numpy.nan])
    assert abs(y[0] - math.exp(700.0)) <= math.ulp(math.exp(700.0))
    assert y[1] == numpy.inf and y[2] == numpy.inf and numpy.isnan(y[3])
