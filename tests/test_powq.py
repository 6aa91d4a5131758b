"""sfx_powq (the plain-FP64 exact solver's quick power, sfx_powq.h) returns
sfx_pow's bits, compiled here from the same sources as the device code."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "shadowfax_b200" / "csrc"

_SRC = r"""
#include "sfx_pow.h"
static long rare;
static double counted(double x, double y) { rare++; return sfx_pow(x, y); }
#define SFX_POWQ_RARE counted
#include "sfx_powq.h"
long differing(const double* x, const double* y, long n, long* slow) {
    long bad = 0;
    rare = 0;
    for(long i = 0; i < n; ++i) {
        const double a = sfx_powq(x[i], y[i]), b = sfx_pow(x[i], y[i]);
        if(sfx_d2u(a) != sfx_d2u(b) && !(a != a && b != b)) ++bad;
    }
    *slow = rare;
    return bad;
}
"""


@pytest.fixture(scope="module")
def differing(tmp_path_factory):
    d = tmp_path_factory.mktemp("powq")
    (d / "q.c").write_text(_SRC)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-mfma", "-shared", "-fPIC", "-I", str(CSRC),
                    str(d / "q.c"), "-o", str(d / "q.so"), "-lm"], check=True)
    fn = C.CDLL(str(d / "q.so")).differing
    fn.restype = C.c_long

    def run(x, y):
        x, y = np.broadcast_arrays(np.asarray(x, np.float64), np.asarray(y, np.float64))
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        slow = C.c_long()
        p = C.POINTER(C.c_double)
        bad = fn(x.ctypes.data_as(p), y.ctypes.data_as(p), C.c_long(x.size), C.byref(slow))
        return bad, slow.value / x.size
    return run


def _exponents(g):
    return [0.5 * (g - 1) / g, -0.5 * (g + 1) / g, 2 / (g - 1), 2 * g / (g - 1), 1 / g]


@pytest.mark.parametrize("gamma", [5 / 3, 1.4])
def test_equal_on_the_solvers_exponents(differing, gamma):
    rng = np.random.default_rng(5)
    n = 300_000
    near = 1 + (rng.random(n) - 0.5) * np.exp(-36 * rng.random(n))
    wide = np.exp(8 * (rng.random(n) - 0.5))
    # both sides of every table interval's edge
    edge = (1 + np.arange(65) / 64)[:, None] * (1 + np.arange(-3, 4) * 2.0**-52)
    for y in _exponents(gamma):
        for x in (near, wide, edge, edge / 2):
            bad, slow = differing(x.ravel(), y)
            assert bad == 0
            if x is wide and abs(y) < 5:   # the rounding test settles all but a few
                assert slow < 1e-3


def test_equal_at_the_range_limit_and_on_special_values(differing):
    rng = np.random.default_rng(6)
    t = 22 + (rng.random(50_000) - 0.5) * 1e-3       # |y ln x| on both sides of 22
    for y in (0.2, -0.8, 3.0):
        assert differing(np.exp(t / y), y)[0] == 0
        assert differing(np.exp(-t / y), y)[0] == 0
    sp = np.array([0.0, -0.0, 1.0, -1.0, 0.5, 2.0, 1e-310, np.inf, -np.inf, np.nan, 4.0, 1e300,
                   1e-300, 3.0, 2.2250738585072014e-308, 1.7976931348623157e308])
    x, y = np.meshgrid(sp, sp)
    assert differing(x.ravel(), y.ravel())[0] == 0
    # exact halfway cases: x^3 of 18-bit integers has 54 bits
    odd = rng.integers(1 << 17, 1 << 18, 50_000) | 1
    assert differing(odd.astype(np.float64), 3.0)[0] == 0
