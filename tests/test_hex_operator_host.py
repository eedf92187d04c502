"""The C3D8 element operator's arithmetic on the host (no GPU): modes stored
and loaded by index as the bricks do, forces against the oracle's element
stiffness."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle
from solvix_b200 import abi

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "solvix_b200", "csrc")

SOURCE = r"""
#include "svx_hex.h"
using namespace svx;
static_assert(sizeof(HexModes) == 21 * sizeof(double) && sizeof(HexModes::c) == sizeof(HexModes),
              "the 21 modes are one array");
extern "C" void element_forces(const double* xyz, const double* u, double E, double nu,
                               double* f) {
    double x[8][3], v[8][3], store[21], rdet[8];
    for (int a = 0; a < 8; ++a)
        for (int c = 0; c < 3; ++c) {
            x[a][c] = xyz[3 * a + c];
            v[a][c] = u[3 * a + c];
        }
    HexModes made(x), X, U(v);
    for (int q = 0; q < 21; ++q) store[q] = made.at(q);
    for (int g = 0; g < 8; ++g) {
        double J[3][3];
        made.gradient(g, J);
        rdet[g] = 1.0 / hex_det(J);
    }
    for (int q = 0; q < 21; ++q) X.at(q) = store[q];
    double lam, mu;
    hex_lame(E, nu, lam, mu);
    HexForces F;
    hex_integrate(X, U, lam, mu, [&](int g) { return rdet[g]; }, F);
    F.nodal(v);
    for (int a = 0; a < 8; ++a)
        for (int c = 0; c < 3; ++c) f[3 * a + c] = v[a][c];
    f[24] = F.work(U);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("hex")
    src, so = d / "hex.cpp", d / "hex.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror",
                    "-Wno-unknown-pragmas", f"-I{CSRC}", str(src), "-o", str(so)], check=True)
    return C.CDLL(str(so))


CORNERS = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0],
                    [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]], float)


@pytest.mark.parametrize("jitter,scale", [(0.0, 1.0), (0.1, 0.0125), (0.2, 7.0)])
def test_forces_are_the_element_stiffness_times_u(lib, jitter, scale):
    rng = np.random.default_rng(int(scale * 80))
    for _ in range(20):
        xyz = scale * (CORNERS + rng.uniform(-jitter, jitter, (8, 3)))
        E, nu = 10.0 ** rng.uniform(9, 11), rng.uniform(0.0, 0.45)
        u, f = rng.standard_normal(24), np.zeros(25)
        p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in (xyz, u, f)]
        lib.element_forces(p[0], p[1], C.c_double(E), C.c_double(nu), p[2])
        reason, ke = oracle.element_stiffness(abi.SVX_C3D8, xyz, E, nu)
        assert reason == 0
        # some 300 roundings of 1.1e-16 lie on the way to a component
        bound = 4e-14 * (np.abs(ke) @ np.abs(u)).max()
        assert np.abs(f[:24] - ke @ u).max() <= bound
        assert abs(f[24] - u @ ke @ u) <= bound * np.abs(u).sum()
