"""The plane PCG's division from a reciprocal, over its range, at its ends and
outside (no GPU)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "solvix_b200", "csrc")

SOURCE = r"""
#include "svx_quotient.h"
extern "C" void quotients(long n, const double* x, const double* y, double* q) {
    for (long k = 0; k < n; ++k) q[k] = svx::quotient(x[k], y[k], 1.0 / y[k]);
}
"""


@pytest.fixture(scope="module")
def quotient(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    f"-I{CSRC}", str(d / "q.cpp"), "-o", str(d / "q.so")], check=True)
    lib = C.CDLL(str(d / "q.so"))
    p = C.POINTER(C.c_double)

    def f(x, y):
        x, y = (np.ascontiguousarray(a, dtype=np.float64).ravel() for a in (x, y))
        q = np.empty_like(x)
        lib.quotients(C.c_long(x.size), *(a.ctypes.data_as(p) for a in (x, y, q)))
        return q
    return f


def pairs(a, b):
    x, y = np.meshgrid(a, b)
    return x.ravel(), y.ravel()


def within_an_ulp(q, x, y):
    with np.errstate(all="ignore"):
        exact = x / y
    assert np.all(np.abs(q - exact) <= np.spacing(np.abs(exact)))


def test_inside_the_range(quotient):
    rng = np.random.default_rng(1)
    n = 400000
    x = rng.uniform(1, 10, n) * 10.0 ** rng.uniform(-139.9, 138.9, n) * rng.choice([-1, 1], n)
    y = rng.uniform(1, 10, n) * 10.0 ** rng.uniform(-139.9, 138.9, n) * rng.choice([-1, 1], n)
    within_an_ulp(quotient(x, y), x, y)
    # the mantissas where a reciprocal is furthest off
    m = np.concatenate([1.0 + np.arange(200) * 2.0 ** -52, 2.0 - np.arange(1, 200) * 2.0 ** -52])
    x, y = pairs(m, m)
    within_an_ulp(quotient(x, y), x, y)


def test_at_the_ends(quotient):
    ends = []
    for e in (1e-140, 1e140):
        for k in range(-40, 41):
            ends.append(e * (1.0 + k * 2.0 ** -52))
    x, y = pairs(ends, ends)
    within_an_ulp(quotient(x, y), x, y)


def test_outside_is_the_division(quotient):
    odd = [0.0, -0.0, 5e-324, 1e-310, 2.3e-308, 1e-200, 9.9e-141, 1.1e140, 1e200, 1.7e308,
           np.inf, -np.inf, np.nan]
    plain = [1.0, -3.0, 1e-139, 1e139]
    for a, b in ((odd, odd), (odd, plain), (plain, odd)):
        x, y = pairs(a, b)
        with np.errstate(all="ignore"):
            np.testing.assert_array_equal(quotient(x, y), x / y)
