"""The fixed-point paths of the correctly rounded log/exp/pow (epic_gb300/csrc/fix_math.cuh) where
they change over: the edges of their tables' intervals, the limits of their arguments, and the
arguments they leave to the double-double evaluation.  Host-compiled (libepicport_cr.so), against
200-bit mpmath evaluations rounded once to binary64."""
import ctypes as C
import math

import numpy as np
import pytest

from oracle_lib import PORT_CR_LIB, build_port

mpmath = pytest.importorskip("mpmath")


@pytest.fixture(scope="module")
def cr():
    build_port()
    lib = C.CDLL(PORT_CR_LIB)
    for n, k in (("log", 1), ("exp", 1), ("pow", 2)):
        f = getattr(lib, "epic_cr_" + n)
        f.restype, f.argtypes = C.c_double, [C.c_double] * k
    return lib


def _around(values, steps=2):
    out = []
    for v in values:
        lo = hi = float(v)
        out.append(lo)
        for _ in range(steps):
            lo, hi = math.nextafter(lo, -math.inf), math.nextafter(hi, math.inf)
            out += [lo, hi]
    return out


# the log table's interval edges 1 + i/1024, over binades, and the smallest normal numbers
EDGES = [math.ldexp(1. + i / 1024., e) for i in range(0, 1024, 31) for e in (-1, 0, 16)] + [1023. / 512., 2.2250738585072014e-308,
                                                                                            1.7976931348623157e308 / 2.]


@pytest.mark.parametrize("what", ["log", "exp", "pow", "special"])
def test_changeovers(cr, what):
    mpmath.mp.prec = 400
    rng = np.random.default_rng(4)
    mp = mpmath.mpf
    if what == "log":
        # around 1: the fixed path serves |log x| >= 2^-12
        xs = _around(EDGES) + _around([1. + s * 2.**-q for q in range(5, 53, 3) for s in (1, -1)])
        bad = [x for x in xs if cr.epic_cr_log(x) != float(mpmath.log(mp(x)))]
    elif what == "exp":
        # the limits 2^-30 and 690, and the intervals of 2^(j/1024)
        xs = _around([s * v for s in (1., -1.) for v in (2.**-31, 2.**-30, 1e-3, 0.5, 689., 690., 699.)])
        xs += _around([j * math.log(2.) / 1024. for j in range(-2100, 2100, 97)], 1) + list(rng.uniform(-700, 700, 500))
        bad = [x for x in xs if cr.epic_cr_exp(x) != float(mpmath.exp(mp(x)))]
    elif what == "pow":
        ys = [2.**-21, 2.**-20, 1. / 6., .25, 2. / 7., 1., 9. / 7., 3.5, 8., 15.999, 16., 17.25]
        xs = _around(EDGES[::5], 1) + list(np.exp(rng.uniform(-12, 12, 40)))
        # |y log2 x| below 1000, results in the normal range
        pairs = [(x, s * y) for x in xs for y in ys for s in (1., -1.) if abs(y * math.log(x)) < 690.]
        bad = [(x, y) for x, y in pairs if cr.epic_cr_pow(x, y) != float(mpmath.power(mp(x), mp(y)))]
    else:
        inf, nan = math.inf, math.nan
        assert cr.epic_cr_log(0.) == -inf and cr.epic_cr_log(inf) == inf and math.isnan(cr.epic_cr_log(-1.))
        assert math.isnan(cr.epic_cr_log(nan)) and cr.epic_cr_log(1.) == 0. and cr.epic_cr_log(5e-324) == math.log(5e-324)
        assert cr.epic_cr_exp(0.) == 1. and cr.epic_cr_exp(-inf) == 0. and cr.epic_cr_exp(inf) == inf and math.isnan(cr.epic_cr_exp(nan))
        assert cr.epic_cr_exp(-745.) == math.exp(-745.)   # a subnormal result
        assert cr.epic_cr_pow(3., 0.) == 1. and cr.epic_cr_pow(1., 1e300) == 1. and cr.epic_cr_pow(0., 3.) == 0.
        assert cr.epic_cr_pow(-3., 3.) == -27. and math.isnan(cr.epic_cr_pow(-3., .5)) and cr.epic_cr_pow(-1.5, 2.) == 2.25
        assert cr.epic_cr_pow(4., .5) == 2. and cr.epic_cr_pow(8., 1. / 3.) == float(mpmath.power(8, mp(1. / 3.)))
        assert math.isnan(cr.epic_cr_pow(nan, 2.)) and math.isnan(cr.epic_cr_pow(2., nan)) and cr.epic_cr_pow(inf, -1.) == 0.
        bad = []
    assert not bad, bad[:5]
