// Fixed-point element operator: K u of an element in 64-bit integers.
//
// GB300 issues about 64 FP32 or integer instructions in the time of one FP64
// one, and most of the modal element operator is additions (the Walsh-Hadamard
// transforms), which are two instructions each, and exact, on 64-bit integers.
// So each displacement is split once per vertex into a signed 57-bit mantissa
// and an exponent, the transforms run on integers, and the few products (22 an
// element) are 64 x 59-bit integer products.
//
// Units and ranges:
//  - an element takes each component of its eight nodes to the largest exponent
//    E_i of that component: |v| <= 2^57, exact for values within four binary
//    orders of the largest, as they are wherever a field is smooth.
//  - its modes are sums of eight of them, |c| <= 2^60, exact.  The components
//    are then brought to a common unit in which the largest mode is just below
//    2^60 (X: its exponent), and the products with rho^p times the modal
//    constants, 59-bit integers of exponent x, come out within 1.25 units, a
//    unit being 2^-57 of that largest mode by the largest constant.
//  - the force is an integer of exponent X + x (fx_to), below 2^63 for any u;
//    each of the three additions that combine the elements of a vertex first
//    halves its operands (fx_down), so no sum can leave 64 bits.
// Everything is relative to the element's own largest mode: a large displacement
// of the void does not blunt a stiff element next to it.  The three components of
// an element share that unit (FP64 would keep a component that is 2^40 smaller,
// and not coupled to the others, to more digits of its own).  Adding forces of
// different exponents shifts the smaller one further, as a floating addition
// would.  Shifts round down.  Displacements below the normal range count as 0,
// and so do forces (the double-float form lost all below 2^-126).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

namespace topo {

constexpr int FX_BAD = 1 << 24;    // exponent of a force that is not a number
constexpr int FX_ZERO = -(1 << 20);  // exponent of no force

// modal constants: lambda h/48, mu h/48, (lambda + 4 mu) h/144
struct FxConst {
  double e, f, g;
};

__host__ __device__ __forceinline__ uint64_t fx_bits(double v) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(v);
#else
  uint64_t b;
  memcpy(&b, &v, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double fx_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}

// u as mantissa times 2^(e - 1079), |mantissa| < 2^57 (below the normal range:
// 0 and e = 0; infinite or not a number: e = 0x7ff)
__host__ __device__ __forceinline__ int64_t fx_split(double u, int& e) {
  const uint64_t b = fx_bits(u);
  e = (int)(b >> 52) & 0x7ff;
  const uint64_t m = e ? ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 4 : 0;
  return (int64_t)((b >> 63) ? 0 - m : m);
}

// y 2^(F - 2098), rounded to nearest (below the normal range: 0)
__host__ __device__ __forceinline__ double fx_to(int64_t y, int F) {
  const uint64_t b = fx_bits((double)y);
  const int e = ((int)(b >> 52) & 0x7ff) + F - 2098;
  if (F >= FX_BAD / 2) return fx_double(0x7ff8000000000000ull);
  if (y == 0 || e <= 0) return 0.0;
  if (e >= 0x7ff) return fx_double((b & 0x8000000000000000ull) | 0x7ff0000000000000ull);
  return fx_double((b & 0x800fffffffffffffull) | ((uint64_t)e << 52));
}

// v 2^k (below the normal range: 0)
__host__ __device__ __forceinline__ double fx_scale(double v, int k) {
  const uint64_t b = fx_bits(v);
  const int e0 = (int)(b >> 52) & 0x7ff, e = e0 + k;
  if (e0 == 0x7ff) return v;
  if (e0 == 0 || e <= 0) return 0.0;
  if (e >= 0x7ff) return fx_double((b & 0x8000000000000000ull) | 0x7ff0000000000000ull);
  return fx_double((b & 0x800fffffffffffffull) | ((uint64_t)e << 52));
}

// p in units of 2^(x - 1081): below 2^59 for exponents up to x
__host__ __device__ __forceinline__ int64_t fx_factor(double p, int x) {
  const uint64_t b = fx_bits(p);
  const int e = (int)(b >> 52) & 0x7ff, k = x - e;
  const uint64_t m = e ? (b & 0xfffffffffffffull) | 0x10000000000000ull : 0;
  const int64_t q = k < 60 ? (int64_t)((m << 6) >> k) : 0;
  return (b >> 63) ? -q : q;
}

// a p / 2^62 for |a| < 2^62, |p| < 2^59, off by -1.25 to 0.75 units and unbiased:
// the product of the low halves is left out (0 to 1 unit, a quarter in the mean,
// which the rounding constant adds back)
__host__ __device__ __forceinline__ int64_t fx_mul(int64_t a, int64_t p) {
  const int ph = (int)(p >> 31), pl = (int)(p & 0x7fffffff);
  const int ah = (int)(a >> 31), al = (int)(a & 0x7fffffff);
  const int64_t m = (int64_t)ah * pl + ((int64_t)al * ph + ((1 << 30) + (1 << 29)));
  return (int64_t)ah * ph + (m >> 31);
}

__host__ __device__ __forceinline__ int fx_clz(unsigned v) {
#ifdef __CUDA_ARCH__
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}

// In: v[3][8] nodal displacements, component i in units of 2^(ei - 1079),
// |v| <= 2^57.  Out: modes 1 to 7 of each component, in units of 2^(X - 1079)
// with the largest just below 2^60; X is returned (FX_ZERO: all zero).
__host__ __device__ __forceinline__ int fx_modes(int64_t v[3][8], int e0, int e1, int e2) {
  int sh[3], X[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    int64_t* q = v[i];
    const int64_t s0 = q[0] + q[1], d0 = q[1] - q[0], s1 = q[2] + q[3], d1 = q[3] - q[2];
    const int64_t s2 = q[4] + q[5], d2 = q[5] - q[4], s3 = q[6] + q[7], d3 = q[7] - q[6];
    const int64_t ss0 = s0 + s1, sd0 = s1 - s0, ds0 = d0 + d1, dd0 = d1 - d0;
    const int64_t ss1 = s2 + s3, sd1 = s3 - s2, ds1 = d2 + d3, dd1 = d3 - d2;
    q[1] = ds0 + ds1; q[2] = sd0 + sd1; q[3] = dd0 + dd1; q[4] = ss1 - ss0;
    q[5] = ds1 - ds0; q[6] = sd1 - sd0; q[7] = dd1 - dd0;
    unsigned top = 0;
#pragma unroll
    for (int m = 1; m < 8; ++m) {
      const int hi = (int)(q[m] >> 32);
      top |= (unsigned)(hi ^ (hi >> 31));
    }
    int lz = fx_clz(top);
    if (top == 0) {  // all modes below 2^32: constant displacement, or nearly
#pragma unroll
      for (int m = 1; m < 8; ++m) top |= (unsigned)(q[m] ^ (q[m] >> 63));
      lz = 32 + fx_clz(top);
    }
    sh[i] = lz > 4 ? lz - 4 : 0;  // largest mode below 2^(64 - lz) -> below 2^60
    X[i] = lz < 64 ? (i == 0 ? e0 : i == 1 ? e1 : e2) - sh[i] : FX_ZERO;
  }
  const int XX = X[0] > X[1] ? (X[0] > X[2] ? X[0] : X[2]) : (X[1] > X[2] ? X[1] : X[2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int r = XX - X[i] < 63 ? XX - X[i] : 63;
#pragma unroll
    for (int m = 1; m < 8; ++m) v[i][m] = (int64_t)((uint64_t)v[i][m] << sh[i]) >> r;
  }
  return XX;
}

// In: v as for fx_modes.  Out: nodal forces, and their exponent is returned.
// The modes and their coefficients are modal_element's (k_fine.cu).
__host__ __device__ __forceinline__ int fx_element(int64_t v[3][8], int e0, int e1, int e2, double pe,
                                                   const FxConst& k) {
  const double pE = pe * k.e, pF = pe * k.f, pG = pe * k.g;
  const int xe = (int)(fx_bits(pE) >> 52) & 0x7ff, xf = (int)(fx_bits(pF) >> 52) & 0x7ff,
            xg = (int)(fx_bits(pG) >> 52) & 0x7ff;
  const int x = xe > xf ? (xe > xg ? xe : xg) : (xf > xg ? xf : xg);
  const int64_t E = fx_factor(pE, x), F = fx_factor(pF, x), G = fx_factor(pG, x);
  const int XX = fx_modes(v, e0, e1, e2);
  int64_t(*c)[8] = v;
  // constant part of the gradient (three times the coefficients of the others)
  const int64_t t = fx_mul(c[0][1] + c[1][2] + c[2][4], E);
  const int64_t sxy = 3 * fx_mul(c[0][2] + c[1][1], F), sxz = 3 * fx_mul(c[0][4] + c[2][1], F),
                syz = 3 * fx_mul(c[1][4] + c[2][2], F);
  const int64_t g01 = 3 * (t + 2 * fx_mul(c[0][1], F)), g12 = 3 * (t + 2 * fx_mul(c[1][2], F)),
                g24 = 3 * (t + 2 * fx_mul(c[2][4], F));
  // X, Y and Z parts
  const int64_t tx = fx_mul(c[1][3] + c[2][5], E), ty = fx_mul(c[0][3] + c[2][6], E), tz = fx_mul(c[0][5] + c[1][6], E);
  const int64_t ryz = fx_mul(c[1][5] + c[2][3], F), rxz = fx_mul(c[0][6] + c[2][3], F),
                rxy = fx_mul(c[0][6] + c[1][5], F);
  const int64_t g03 = 3 * fx_mul(c[0][3], F) + ty, g13 = 3 * fx_mul(c[1][3], F) + tx, g23 = ryz + rxz;
  const int64_t g05 = 3 * fx_mul(c[0][5], F) + tz, g15 = ryz + rxy, g25 = 3 * fx_mul(c[2][5], F) + tx;
  const int64_t g06 = rxz + rxy, g16 = 3 * fx_mul(c[1][6], F) + tz, g26 = 3 * fx_mul(c[2][6], F) + ty;
  const int64_t g07 = fx_mul(c[0][7], G), g17 = fx_mul(c[1][7], G), g27 = fx_mul(c[2][7], G);
  const int64_t g[3][8] = {{0, g01, sxy, g03, sxz, g05, g06, g07},
                           {0, sxy, g12, g13, syz, g15, g16, g17},
                           {0, sxz, syz, g23, g24, g25, g26, g27}};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int zb = 0; zb < 2; ++zb) {
      const int64_t h0 = zb ? g[i][4] : -g[i][4], h1 = zb ? g[i][1] + g[i][5] : g[i][1] - g[i][5];
      const int64_t h2 = zb ? g[i][2] + g[i][6] : g[i][2] - g[i][6], h3 = zb ? g[i][3] + g[i][7] : g[i][3] - g[i][7];
      const int64_t a0 = h0 - h2, a1 = h1 - h3, b0 = h0 + h2, b1 = h1 + h3;
      v[i][4 * zb] = a0 - a1; v[i][4 * zb + 1] = a0 + a1;
      v[i][4 * zb + 2] = b0 - b1; v[i][4 * zb + 3] = b0 + b1;
    }
  }
  return XX + x;
}

// a shifted right by k >= 0
__host__ __device__ __forceinline__ int64_t fx_down(int64_t a, int k) { return a >> (k < 63 ? k : 63); }

}  // namespace topo
