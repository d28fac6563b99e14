// The FP64 fine operator of the CG solvers in 64-bit fixed point (fx.cuh): K u,
// f - K u and the FP64 Chebyshev step on level 0.
//
// Bound and layout.  The z march, tiles, z blocks and void narrowing are those
// of k_fine_modal.  What bounds the FP64 form is the FP64 pipe (240 operations
// an element, two lanes a clock and SM), what bounds the double-float form is
// about 3,000 FP32 instructions an element; this form needs about 1,000 integer
// instructions an element and 6 to 20 FP64 operations a vertex (conversions and
// the Chebyshev update), which run beside each other.
// Its error is below the FP64 kernel's: the transforms are exact and only the
// 22 products of an element round.
//
// Per step (element layer ez), one barrier:
//   before it each thread splits its staged vertices of plane ez + 1 into
//     mantissas and exponents, into a slot of three that no thread of the step
//     before reads (it stages and converts the same vertices, so their copies
//     need no barrier);
//   after it, with plane ez + 1 converted and the last layer's y = 0 forces
//     published, it finishes its vertex of plane ez - 1 from the two layers next
//     to it and computes its element: the FP64 chain of the one and the integer
//     work of the other are in one phase, where the 16 warps of an SM fill each
//     other's gaps.
// With a barrier on either side of the vertex, and two converted planes, the
// Chebyshev step at 128x64x64 took 100.9 us (now 97.9), K u 67.6 (66.1): issue
// slots 45% busy there, the FP64 pipe 31%, a sixth of the stalls at barriers.
#include "topo_internal.h"

#include "fx.cuh"

namespace topo {

__constant__ FxConst cFx;

void upload_fx(double lam, double mu, double h) {
  const FxConst c{lam * h / 48.0, mu * h / 48.0, (lam + 4.0 * mu) * h / 144.0};
  cudaMemcpyToSymbol(cFx, &c, sizeof(c));
}

namespace {

constexpr int FX_CTAS = 2;  // resident on an SM (128 registers a thread)
constexpr int TX = FINE_TILE_X, TY = FINE_TILE_Y, NT = TX * TY, PX = TX + 1, NP = PX * (TY + 1);
constexpr int KS = (NP + NT - 1) / NT;  // vertices of a plane a thread stages

struct FxSmem {
  longlong2 qa[3][NP];     // converted planes: mantissas of components 0 and 1
  longlong2 qb[3][NP];     //                   of component 2, exponents (16 bits each)
  double raw[3][3][NP];    // staged planes
  longlong2 xa[2][3][NT];  // y = 0 forces of a layer: z = 0 (c0, c1), (c2, z = 1 c0), z = 1 (c1, c2)
  int xe[2][NT];           // their exponent
};

__device__ __forceinline__ void stage8(double* smem, const double* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 8 : 0));
}

// Arguments of the Chebyshev step (MODE 2): r = f - K u, d = c_old d + c_new
// D^-1 r (first: c_new D^-1 r), out = u + d.
struct FxCheb {
  const double* dinv;  // [9][nv]
  double* dvec;        // [3][nv]
  const double* coef;  // (c_old, c_new)
  int first;
};

// MODE 0: out = K u, 1: out = f - K u, 2: Chebyshev step
template <int MODE, bool VOID>
__global__ void __launch_bounds__(NT, FX_CTAS) k_fine_fx(LevelDims d, const double* __restrict__ rhop,
                                                   const uint8_t* __restrict__ vmask, const double* __restrict__ u,
                                                   const double* __restrict__ f, double* __restrict__ out, ZSplit zs,
                                                   FxCheb ch) {
  extern __shared__ __align__(16) unsigned char fx_smem[];
  FxSmem& sm = *reinterpret_cast<FxSmem*>(fx_smem);
  const int t = threadIdx.x, i = t % TX, j = t / TX;
  const int rhs = blockIdx.z / zs.n, kz = blockIdx.z - rhs * zs.n;
  const int x0 = blockIdx.x * (TX - 1), y0 = blockIdx.y * (TY - 1), zb0 = zs.begin(kz);
  const int64_t nv = d.nv, plane_n = (int64_t)d.vx * d.vy;
  u += (int64_t)rhs * 3 * nv;
  if (MODE >= 1) f += (int64_t)rhs * 3 * nv;
  out += (int64_t)rhs * 3 * nv;
  double* __restrict__ dv = MODE == 2 ? ch.dvec + (int64_t)rhs * 3 * nv : nullptr;
  const int gx = x0 + i, gy = y0 + j;  // owned vertex (x, y) and element (x - 1, y - 1)
  const bool own = i < TX - 1 && j < TY - 1 && gx < d.vx && gy < d.vy;
  const int zb1 = zs.end(kz, zb0);
  int z0 = zb0, zend = zb1;  // the planes marched: [zb0, zb1) less the void (LevelDims::colz)
  if (VOID) {
    const int2 cz = d.colz[blockIdx.x + gridDim.x * blockIdx.y];
    z0 = min(max(zb0, cz.x), zb1);
    zend = max(z0, min(zb1, cz.y + 2));
  }
  // What the owned vertex of plane p needs besides its element forces.  Loaded
  // before the step's barrier, so that the loads' latency passes there.
  struct Vertex {
    int64_t v;
    uint8_t m;
    double f[3], di[MODE == 2 ? 9 : 1], d[3], u[3];
  };
  auto load_vertex = [&](int p, Vertex& V) {
    V.v = gx + (int64_t)d.vx * gy + plane_n * p;
    V.m = vmask[V.v];
    if (MODE >= 1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) V.f[c] = f[c * nv + V.v];
    }
    if (MODE == 2) {
#pragma unroll
      for (int c = 0; c < 9; ++c) V.di[c] = ch.dinv[c * nv + V.v];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        V.d[c] = ch.first ? 0.0 : dv[c * nv + V.v];
        V.u[c] = u[c * nv + V.v];
      }
    }
  };
  // the vertex with its element forces y (fixed DOFs: none)
  auto finish = [&](const Vertex& V, const double y[3]) {
    if (MODE < 2) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const bool fr = (V.m >> c) & 1;
        out[c * nv + V.v] = MODE == 1 ? (fr ? V.f[c] - y[c] : 0.0) : (fr ? y[c] : 0.0);
      }
    } else {
      double r[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) r[c] = ((V.m >> c) & 1) ? V.f[c] - y[c] : 0.0;
      const double c_old = __ldg(ch.coef), c_new = __ldg(ch.coef + 1);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double z = V.di[3 * c] * r[0] + V.di[3 * c + 1] * r[1] + V.di[3 * c + 2] * r[2];
        const double dn = ch.first ? c_new * z : c_old * V.d[c] + c_new * z;
        dv[c * nv + V.v] = dn;
        out[c * nv + V.v] = V.u[c] + dn;
      }
    }
  };
  if (VOID && own) {  // void planes see no forces
    const double none[3] = {0.0, 0.0, 0.0};
    Vertex V;
    for (int p = zb0; p < z0; ++p) { load_vertex(p, V); finish(V, none); }
    for (int p = zend; p < zb1; ++p) { load_vertex(p, V); finish(V, none); }
  }
  if (z0 >= zend) return;  // the whole CTA
  int pxy[KS];  // this thread's staged vertices, in-plane (-1: outside the domain)
#pragma unroll
  for (int s = 0; s < KS; ++s) {
    const int k = t + s * NT, px = k % PX, py = k / PX, vx = x0 - 1 + px, vy = y0 - 1 + py;
    pxy[s] = (k < NP && vx >= 0 && vy >= 0 && vx < d.vx && vy < d.vy) ? vx + d.vx * vy : -1;
  }
  auto prefetch = [&](int z) {
    if (z <= zend) {
      double(*dst)[NP] = sm.raw[(z + 3) % 3];
      const bool zok = z >= 0 && z < d.vz;
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const int k = t + s * NT;
        if (k < NP) {
          const bool ok = zok && pxy[s] >= 0;
          const double* src = u + (ok ? plane_n * z + pxy[s] : 0);
          stage8(&dst[0][k], src, ok);
          stage8(&dst[1][k], src + nv, ok);
          stage8(&dst[2][k], src + 2 * nv, ok);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  auto convert = [&](int z) {
    const double(*src)[NP] = sm.raw[(z + 3) % 3];
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      const int k = t + s * NT;
      if (k < NP) {
        int e0, e1, e2;
        const int64_t q0 = fx_split(src[0][k], e0), q1 = fx_split(src[1][k], e1), q2 = fx_split(src[2][k], e2);
        sm.qa[(z + 3) % 3][k] = make_longlong2(q0, q1);
        sm.qb[(z + 3) % 3][k] = make_longlong2(q2, (long long)((uint64_t)(unsigned)(e0 | e1 << 16) | (uint64_t)e2 << 32));
      }
    }
  };
  const int ex = gx - 1, ey = gy - 1;
  const bool pe_xy = ex >= 0 && ey >= 0 && ex < d.ex && ey < d.ey;
  auto load_pe = [&](int ez) -> double {
    return (pe_xy && ez >= 0 && ez < d.ez) ? rhop[ex + (int64_t)d.ex * (ey + (int64_t)d.ey * ez)] : 0.0;
  };
  int64_t own1[2][3] = {{0, 0, 0}, {0, 0, 0}}, top[3] = {0, 0, 0};  // y = 1 forces of the last layer; z = 1 of the one below
  int oe = FX_ZERO, te = FX_ZERO;  // their exponents
  prefetch(z0 - 1);
  prefetch(z0);
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  convert(z0 - 1);
  double pe_n = load_pe(z0 - 1);
  // step st: finish vertex plane st - 1 (layers st - 2 and st - 1), compute element layer st
  for (int st = z0 - 1; st <= zend; ++st) {
    const double pe = pe_n;
    Vertex V;
    if (st - 1 >= z0 && own) load_vertex(st - 1, V);
    if (st < zend) {
      prefetch(st + 2);
      if (st + 1 < zend) pe_n = load_pe(st + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // plane st + 1 has arrived
    }
    if (st < zend) convert(st + 1);
    __syncthreads();
    if (st >= z0 && own) {
      const int xs = (st - 1) & 1, n = t + TX;
      const longlong2 a = sm.xa[xs][0][n], b = sm.xa[xs][1][n], c2 = sm.xa[xs][2][n];
      const int re = sm.xe[xs][n], ye = max(oe, re);
      const int64_t r0[3] = {a.x, a.y, b.x}, r1[3] = {b.y, c2.x, c2.y};
      const int ze = max(te, ye + 1);
      double y[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t bot = fx_down(own1[0][c], ye - oe + 1) + fx_down(r0[c], ye - re + 1);
        y[c] = fx_to(fx_down(top[c], ze - te + 1) + fx_down(bot, ze - ye), ze + 1);
        top[c] = fx_down(own1[1][c], ye - oe + 1) + fx_down(r1[c], ye - re + 1);
      }
      te = ye + 1;
      if (st - 1 >= z0) finish(V, y);
    }
    if (st == zend) break;
    {
      int64_t v[3][8];
      int fe = FX_ZERO;
      if (pe != 0.0) {
        unsigned e01[8], m01 = 0;
        int e2[8], m2 = 0;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const int k = (i + (a & 1)) + PX * (j + ((a >> 1) & 1)), z = (st + 3 + (a >> 2)) % 3;
          const longlong2 p = sm.qa[z][k], q = sm.qb[z][k];
          v[0][a] = p.x; v[1][a] = p.y; v[2][a] = q.x;
          e01[a] = (unsigned)q.y;
          e2[a] = (int)(q.y >> 32);
          m01 = __vmaxu2(m01, e01[a]);
          m2 = max(m2, e2[a]);
        }
#pragma unroll
        for (int a = 0; a < 8; ++a) {  // to the element's exponent of each component
          const unsigned k01 = __vminu2(__vsub2(m01, e01[a]), 0x003f003fu);
          v[0][a] >>= k01 & 0xffff;
          v[1][a] >>= k01 >> 16;
          v[2][a] >>= min(m2 - e2[a], 63);
        }
        const int E0 = (int)(m01 & 0xffff), E1 = (int)(m01 >> 16);
        const bool bad = max(max(E0, E1), m2) >= 0x7ff || ((__double2hiint(pe) >> 20) & 0x7ff) == 0x7ff;
        fe = fx_element(v, E0, E1, m2, pe, cFx);
        if (bad) fe = FX_BAD;
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int a = 0; a < 8; ++a) v[c][a] = 0;
      }
      // vertex column i: the x = 1 nodes of element i and the x = 0 nodes of
      // element i + 1 (lane 31's column is not owned), each halved
      const int el = __shfl_up_sync(0xffffffffu, fe, 1), er = __shfl_down_sync(0xffffffffu, fe, 1);
      const int k0 = max(i > 0 ? el - fe : 0, 0) + 1, k1 = max(i < TX - 1 ? er - fe : 0, 0) + 1;
      oe = fe + k1;
      int64_t xc[2][2][3];  // [y][z][component]
#pragma unroll
      for (int yb = 0; yb < 2; ++yb)
#pragma unroll
        for (int zb = 0; zb < 2; ++zb)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int64_t lo = fx_down(v[c][2 * yb + 4 * zb], k0);
            xc[yb][zb][c] = fx_down(v[c][1 + 2 * yb + 4 * zb], k1) + __shfl_down_sync(0xffffffffu, lo, 1);
          }
#pragma unroll
      for (int zb = 0; zb < 2; ++zb)
#pragma unroll
        for (int c = 0; c < 3; ++c) own1[zb][c] = xc[1][zb][c];
      const int xs = st & 1;
      sm.xa[xs][0][t] = make_longlong2(xc[0][0][0], xc[0][0][1]);
      sm.xa[xs][1][t] = make_longlong2(xc[0][0][2], xc[0][1][0]);
      sm.xa[xs][2][t] = make_longlong2(xc[0][1][1], xc[0][1][2]);
      sm.xe[xs][t] = oe;
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

template <int MODE>
void launch(cudaStream_t s, const LevelDims& d, const double* rhop, const uint8_t* vmask, const double* u,
            const double* f, double* out, int nb, int tz, const FxCheb& ch) {
  static PerDeviceOnce once[2];
  const bool vd = d.colz && d.colz_void;
  auto fn = vd ? k_fine_fx<MODE, true> : k_fine_fx<MODE, false>;
  once_per_device(once[vd ? 1 : 0], [&]() -> cudaError_t {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FxSmem));
  });
  const int gx = (d.vx + TX - 2) / (TX - 1), gy = (d.vy + TY - 2) / (TY - 1);
  const ZSplit zs(d.vz, fine_zblocks(d.vz, tz > 0 ? tz : 16, (int64_t)gx * gy * nb, FX_CTAS));
  fn<<<dim3(gx, gy, zs.n * nb), NT, sizeof(FxSmem), s>>>(d, rhop, vmask, u, f, out, zs, ch);
}

}  // namespace

void launch_fine_apply_fx(cudaStream_t s, const LevelDims& d, const double* rhop, const uint8_t* vmask,
                          const double* u, const double* f, double* out, bool residual, int nb, int tz) {
  if (residual) launch<1>(s, d, rhop, vmask, u, f, out, nb, tz, FxCheb{});
  else launch<0>(s, d, rhop, vmask, u, f, out, nb, tz, FxCheb{});
}

void launch_fine_cheb_fx(cudaStream_t s, const LevelDims& d, const double* rhop, const uint8_t* vmask,
                         const double* u, const double* f, double* uout, const double* dinv, double* dvec,
                         const double* coef, bool first, int nb, int tz) {
  launch<2>(s, d, rhop, vmask, u, f, uout, nb, tz, FxCheb{dinv, dvec, coef, first ? 1 : 0});
}

}  // namespace topo
