"""The gradient kernel's division by a stored reciprocal (sfx_div_by, compiled here from the
device code's source) against the division, over the whole range the kernel admits: divisors
between 2^-200 and 2^200, dividends 0 or between 2^-560 and 2^520."""
import ctypes as C
import subprocess

import numpy as np

from test_fp64_gradient_identities import CSRC

_SRC = r"""
#include <stdbool.h>
#include "sfx_limiter.h"
long differing(const double* a, const double* b, long n) {
    long bad = 0;
    for(long i = 0; i < n; ++i) bad += sfx_div_by(a[i], b[i], 1. / b[i]) != a[i] / b[i];
    return bad;
}
"""


def test_equals_the_division(tmp_path):
    (tmp_path / "d.c").write_text(_SRC)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-mfma", "-shared", "-fPIC", "-I", str(CSRC),
                    str(tmp_path / "d.c"), "-o", str(tmp_path / "d.so"), "-lm"], check=True)
    fn = C.CDLL(str(tmp_path / "d.so")).differing
    fn.restype = C.c_long

    def bad(a, b):
        a, b = (np.ascontiguousarray(v, np.float64) for v in np.broadcast_arrays(a, b))
        p = C.POINTER(C.c_double)
        return fn(a.ctypes.data_as(p), b.ctypes.data_as(p), C.c_long(a.size))

    rng = np.random.default_rng(12)
    n = 2_000_000
    b = np.ldexp(1 + rng.random(n), rng.integers(-200, 200, n))
    a = np.ldexp(1 + rng.random(n), rng.integers(-560, 520, n)) * rng.choice([-1, 1], n)
    assert bad(a, b) == 0
    q = 1 + rng.random(n)
    assert bad(q * b, b) == 0 and bad(np.nextafter(q * b, 0), b) == 0   # next to representable ones
    # the ends of the ranges, and mantissas of all ones
    edge_a = np.array([0.0, 2.0**-560, -2.0**520, 2.0**-552, np.nextafter(2.0**520, 0)])
    edge_b = np.array([2.0**-200, 2.0**200, np.nextafter(2.0**-199, 0), np.nextafter(2.0, 0), 1.0])
    m = np.nextafter(np.ldexp(1.0, rng.integers(-199, 200, n)), 0)
    assert bad(edge_a[:, None], edge_b) == 0 and bad(a, m) == 0
