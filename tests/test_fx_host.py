"""The fixed-point arithmetic of the FP64 fine operator (csrc/fx.cuh) on the host: its product against 128-bit integers,
an element's nodal forces against extended precision."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from topoptspline3d_gb300 import build

SOURCE = r"""
#include "fx.cuh"
using namespace topo;
extern "C" void products(const int64_t* a, const int64_t* p, double* err, int n) {
  for (int i = 0; i < n; ++i) {
    const __int128 d = ((__int128)fx_mul(a[i], p[i]) << 62) - (__int128)a[i] * p[i];
    err[i] = (double)d / 0x1p62;
  }
}
// error of the nodal forces of one element, in units of the last place of its force
extern "C" void element(const double* u, double pe, double E, double F, double G, double* err) {
  typedef long double L;
  int64_t v[3][8];
  int e[3] = {0, 0, 0};
  for (int i = 0; i < 3; ++i) {
    int ei[8];
    for (int a = 0; a < 8; ++a) {
      v[i][a] = fx_split(u[8 * i + a], ei[a]);
      e[i] = ei[a] > e[i] ? ei[a] : e[i];
    }
    for (int a = 0; a < 8; ++a) v[i][a] = fx_down(v[i][a], e[i] - ei[a]);
  }
  const FxConst k{E, F, G};
  const int X = fx_element(v, e[0], e[1], e[2], pe, k);
  L c[3][8], g[3][8] = {};
  for (int i = 0; i < 3; ++i) {
    for (int a = 0; a < 8; ++a) c[i][a] = u[8 * i + a];
    for (int h = 1; h < 8; h <<= 1)
      for (int a = 0; a < 8; ++a)
        if (!(a & h)) { const L s = c[i][a], t = c[i][a | h]; c[i][a] = s + t; c[i][a | h] = t - s; }
  }
  const double pE = pe * E, pF = pe * F, pG = pe * G;
  // gradient restricted to each of the functions 1, X, Y, Z, YZ, XZ, XY: (set, weight)
  const int sets[7] = {0, 1, 2, 4, 3, 5, 6};
  for (int q = 0; q < 7; ++q) {
    const int m = sets[q], bits = (m & 1) + (m >> 1 & 1) + (m >> 2);
    // weights 3, 1, 1/3 of lambda h/48 and mu h/48; the last function's constant is G (lambda + 4 mu) h/144 where a
    // component meets all three of them, put in below
    if (bits == 2) continue;
    const L w = bits == 0 ? 3 : 1;
    L D[3][3], tr = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) D[i][j] = m >> j & 1 ? 0 : c[i][m | 1 << j];
    for (int i = 0; i < 3; ++i) tr += D[i][i];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j)
        if (!(m >> j & 1)) g[i][m | 1 << j] += w * ((L)pF * (D[i][j] + D[j][i]) + (i == j ? (L)pE * tr : 0));
  }
  for (int i = 0; i < 3; ++i) g[i][7] = (L)pG * c[i][7];
  for (int i = 0; i < 3; ++i) {
    for (int h = 1; h < 8; h <<= 1)
      for (int a = 0; a < 8; ++a)
        if (!(a & h)) { const L s = g[i][a], t = g[i][a | h]; g[i][a] = s - t; g[i][a | h] = s + t; }
    for (int a = 0; a < 8; ++a) err[8 * i + a] = (double)((L)v[i][a] - ldexpl(g[i][a], 2098 - X));
  }
}
"""


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    (d / "fx.cpp").write_text("#include <math.h>\n" + SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I" + build.CSRC, "-I" + cuda,
                    str(d / "fx.cpp"), "-o", str(d / "fx.so")], check=True)
    return ctypes.CDLL(str(d / "fx.so"))


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_product_within_its_bound_and_without_bias(fx):
    """The dropped product of the low halves is 0 to 1 unit, a quarter in the mean, which the rounding constant puts
    back: -1.25 to 0.75.  A million errors of at most 1.25: four standard errors of their mean are below 0.005."""
    rng = np.random.default_rng(1)
    n = 1000000
    a = rng.integers(-(1 << 62) + 1, 1 << 62, n)
    p = rng.integers(-(1 << 59) + 1, 1 << 59, n)
    a[:6], p[:6] = [0, 5, (1 << 62) - 1, -(1 << 62) + 1, 0, 1], [7, 0, (1 << 59) - 1, (1 << 59) - 1, -7, 1]
    err = np.zeros(n)
    fx.products(_p(a), _p(p), _p(err), n)
    assert err.min() >= -1.25 and err.max() <= 0.75
    assert abs(err.mean()) < 0.005
    assert err[0] == err[1] == err[4] == 0  # zero stays zero


@pytest.mark.parametrize("field", ["rough", "smooth", "one component", "spread"])
@pytest.mark.parametrize("nu", [-0.9, 0.0, 0.4, 0.4999])
def test_element_forces(fx, nu, field):
    """A product is off by 1.25 units and a quarter from the constant's 59 bits, a mode by one unit from the common
    exponent and one from its own (an eighth each after the product); a nodal force adds up to seven modes with up to
    nine products each: 7 x 9 x 1.75 < 111 units, of which a force has up to 2^63."""
    fx.element.argtypes = [ctypes.c_void_p] + [ctypes.c_double] * 4 + [ctypes.c_void_p]
    rng = np.random.default_rng(2)
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)) * 1e6, 1e6 / (2 * (1 + nu))
    err = np.zeros(24)
    worst = 0.0
    for _ in range(2000):
        u = rng.standard_normal((3, 8))
        if field == "smooth":
            u = 1.0 + 1e-4 * u
        elif field == "one component":
            u[1:] *= 1e-9
        elif field == "spread":
            u *= 10.0 ** rng.uniform(-12, 0, (3, 8))
        u = np.ascontiguousarray(u * 10.0 ** rng.uniform(-12, 3))
        fx.element(_p(u), 10.0 ** rng.uniform(-9, 0), lam / 48, mu / 48, (lam + 4 * mu) / 144, _p(err))
        worst = max(worst, float(np.abs(err).max()))
    assert worst < 111
