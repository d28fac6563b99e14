// Design-chain kernels: B-spline density, element sensitivity, sensitivity
// filter, spline adjoint and the OC coefficient trial.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "df.cuh"
#include "fx.cuh"
#include "topo_internal.h"

namespace topo {

static inline unsigned nblk(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

constexpr int MAX_ORDER = 4;  // highest spline order (cubic B-splines)

// v^p for the SIMP exponent: repeated products for small integer p (the
// reference default p = 3), the general pow otherwise.
__device__ __forceinline__ double simp_pow(double v, double p) {
  const int ip = (int)p;
  if ((double)ip == p && ip >= 0 && ip <= 8) {
    double r = 1.0;
    for (int k = 0; k < ip; ++k) r *= v;
    return r;
  }
  return pow(v, p);
}

constexpr int VOL_THREADS = 256;
constexpr int VOL_BLOCKS = 2048;  // partial sums of a trial volume

// End of a trial volume: the CTA's FP64 sum r of its threads' values becomes a
// partial, and the CTA with the last ticket adds the nb partials (in an order
// that does not depend on which CTA is last) into *out and, in a device-side
// bisection, takes the bracket's step.  Done here it costs the trial neither a
// one-CTA kernel nor a one-thread one.  Every thread calls it.
__device__ __forceinline__ void finish_volume(double s, double* partial, double* out, unsigned* ctr, const OcStep& st) {
  __shared__ double ws[32];
  __shared__ bool last;
  const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto cta_sum = [&](double v) {  // valid in thread 0
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) ws[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
      for (int q = 0; q < nw; ++q) r += ws[q];
    return r;
  };
  const double r = cta_sum(s);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = r;
    __threadfence();
    last = atomicAdd(ctr, 1u) == gridDim.x - 1;
    if (last) __threadfence();
  }
  __syncthreads();
  if (!last) return;
  double t = 0.0;
  for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) t += __ldcg(partial + q);
  t = cta_sum(t);
  if (threadIdx.x == 0) {
    *out = t;
    *ctr = 0u;
    if (st.oc) oc_step(st, t);
  }
}

// Separable evaluation, pass 1: B[z][y][i] = sum_{s,t} c[i, iy+s, iz+t] Ny[y][s] Nz[z][t]
// for every x-basis index i (0 where y or z is outside the spline range), in
// FP64, stored split into (hi, lo) floats for the double-float pass 2.
__global__ void k_spline_yz(LevelDims d, SplineDev sp, const double* __restrict__ coeff,
                            float2* __restrict__ B) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nbx = sp.nb[0];
  if (gid >= (int64_t)nbx * d.ey * d.ez) return;
  const int i = (int)(gid % nbx);
  const int64_t yz = gid / nbx;
  const int y = (int)(yz % d.ey), z = (int)(yz / d.ey);
  const int iy = sp.i0[1][y], iz = sp.i0[2][z];
  double v = 0.0;
  if (iy >= 0 && iz >= 0) {
    const int k = sp.order;
    for (int s = 0; s < k; ++s) {
      const double ns = sp.N[1][y * k + s];
      double a = 0.0;
      for (int t = 0; t < k; ++t)
        a += coeff[i + (int64_t)nbx * ((iy + s) + (int64_t)sp.nb[1] * (iz + t))] * sp.N[2][z * k + t];
      v += ns * a;
    }
  }
  const df vd = df_from(v);
  B[gid] = make_float2(vd.hi, vd.lo);
}

// Pass 1 of an OC trial in double-float, from coefficients already split into
// (hi, lo) floats (FP64 here would be bound by the FP64 pipe on every trial).
__global__ void k_spline_yz_df(LevelDims d, SplineDev sp, const float2* __restrict__ coeff,
                               float2* __restrict__ B) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nbx = sp.nb[0];
  if (gid >= (int64_t)nbx * d.ey * d.ez) return;
  const int i = (int)(gid % nbx);
  const int64_t yz = gid / nbx;
  const int y = (int)(yz % d.ey), z = (int)(yz / d.ey);
  const int iy = sp.i0[1][y], iz = sp.i0[2][z];
  df v(0);
  if (iy >= 0 && iz >= 0) {
    const int k = sp.order;
    for (int s2 = 0; s2 < k; ++s2) {
      const float2 ns = sp.Ndf[1][y * k + s2];
      df a(0);
      for (int t = 0; t < k; ++t) {
        const float2 c = coeff[i + (int64_t)nbx * ((iy + s2) + (int64_t)sp.nb[1] * (iz + t))];
        const float2 nz = sp.Ndf[2][z * k + t];
        a += df(c.x, c.y) * df(nz.x, nz.y);
      }
      v += df(ns.x, ns.y) * a;
    }
  }
  B[gid] = make_float2(v.hi, v.lo);
}

// Pass 2: value at element (x,y,z) = sum_r Nx[x][r] B[z][y][ix + r], or -0.2 out of
// range, in double-float arithmetic (about 1e-15 relative; FP64 here would be
// bound by GB300's FP64 pipe, and each OC bisection trial evaluates it on every
// element).
__device__ __forceinline__ df spline_from_B(const SplineDev& sp, const float2* __restrict__ B,
                                            int x, int y, int z, int ey) {
  const int ix = sp.i0[0][x];
  if (ix < 0 || sp.i0[1][y] < 0 || sp.i0[2][z] < 0) return df_from(-0.2);
  const int k = sp.order;
  const float2* b = B + (int64_t)sp.nb[0] * (y + (int64_t)ey * z) + ix;
  df v(0);
  for (int r = 0; r < k; ++r) {
    const float2 n = sp.Ndf[0][x * k + r], bb = b[r];
    v += df(n.x, n.y) * df(bb.x, bb.y);
  }
  return v;
}

// (x, y, z) of element e, in 32-bit arithmetic when the grid allows
__device__ __forceinline__ void elem_xyz(const LevelDims& d, int64_t e, int& x, int& y, int& z) {
  if (d.ne < (int64_t)1 << 31) {
    const unsigned ee = (unsigned)e, ex = (unsigned)d.ex, t = ee / ex;
    x = (int)(ee - t * ex);
    y = (int)(t % (unsigned)d.ey);
    z = (int)(t / (unsigned)d.ey);
  } else {
    x = (int)(e % d.ex);
    const int64_t t = e / d.ex;
    y = (int)(t % d.ey);
    z = (int)(t / d.ey);
  }
}

__device__ __forceinline__ bool df_lt(df a, df b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }

__global__ void k_density_from_B(LevelDims d, const uint8_t* __restrict__ eactive, SplineDev sp,
                                 const float2* __restrict__ B, double rho_min, double penal,
                                 double* __restrict__ rho, double* __restrict__ rhop, float* __restrict__ rhop32) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.ne) return;
  if (!eactive[e]) {
    rho[e] = 0.0; rhop[e] = 0.0; rhop32[e] = 0.0f;
    return;
  }
  int x, y, z;
  elem_xyz(d, e, x, y, z);
  const double v = fmin(fmax(df_to(spline_from_B(sp, B, x, y, z, d.ey)), rho_min), 1.0);
  const double vp = simp_pow(v, penal);
  rho[e] = v; rhop[e] = vp; rhop32[e] = (float)vp;
}

__global__ void __launch_bounds__(VOL_THREADS) k_volume_from_B(LevelDims d, const uint8_t* __restrict__ eactive,
                                                               SplineDev sp, const float2* __restrict__ B,
                                                               double rho_min, double* partial, double* out,
                                                               unsigned* ctr, OcStep st) {
  const df lo = df_from(rho_min), one(1.f, 0.f);
  df sd(0);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < d.ne; e += (int64_t)gridDim.x * blockDim.x) {
    if (!eactive[e]) continue;
    int x, y, z;
    elem_xyz(d, e, x, y, z);
    df v = spline_from_B(sp, B, x, y, z, d.ey);
    if (df_lt(v, lo)) v = lo;
    if (df_lt(one, v)) v = one;
    sd += v;
  }
  finish_volume(df_to(sd), partial, out, ctr, st);
}

// (hi, lo) float split of n doubles
__global__ void k_to_df(int64_t n, const double* __restrict__ a, float2* __restrict__ b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const df v = df_from(a[i]);
  b[i] = make_float2(v.hi, v.lo);
}

// Both passes for a chunk of element rows in one CTA, in double-float.  A chunk
// is up to ych rows y of an element layer z.  C[j][i] = sum_t c[i, j, iz+t]
// Nz[z][t] for the y-basis indices j the rows use and then B[y][i] = sum_s
// Ny[y][s] C[iy+s][i] go to shared memory (the products and their order are
// those of k_spline_yz_df: inner sum over t, outer over s), and each thread
// evaluates its element column x on the chunk's rows with the column's basis
// index and weights in registers (values as spline_from_B).  The table C holds
// cap_j y-basis rows; a chunk whose rows use more (a spline partition finer
// than the elements) forms B straight from the coefficients.
// B never goes to global memory and the two passes are one launch.  A trial
// volume is bound by latency at small grids and by the double-float chains of
// a few rows per thread at large ones: the rows of a chunk are independent, so
// four of them are in flight per thread, with no barrier between rows.
constexpr int ROW_MAX = 1024;  // elements of a row, one thread each
constexpr int CHUNK_Y = 16;    // most rows of a chunk (a warp holds their y-basis indices)
// CTAs aimed at by shortening the chunks of small grids: four on each SM
constexpr int CHUNK_CTAS = 608;
constexpr size_t CHUNK_SMEM = 200 * 1024;  // most shared memory of a CTA's tables

template <int K>
__device__ __forceinline__ df spline_yz_at(const LevelDims& d, const SplineDev& sp, const float2* __restrict__ coeff,
                                           int i, int y, int iz, const df* nz) {
  const int iy = sp.i0[1][y], nbx = sp.nb[0];
  df v(0);
  if (iy < 0) return v;
  for (int s2 = 0; s2 < K; ++s2) {
    const float2 ns = sp.Ndf[1][y * K + s2];
    df a(0);
#pragma unroll
    for (int t = 0; t < K; ++t) {
      const float2 c = coeff[i + (int64_t)nbx * ((iy + s2) + (int64_t)sp.nb[1] * (iz + t))];
      a += df(c.x, c.y) * nz[t];
    }
    v += df(ns.x, ns.y) * a;
  }
  return v;
}

// MODE 0: volume of the clamped values of active elements (partial, *out, st);
// MODE 1: densities rho, rho^p (FP64 and FP32) of every element.
// K: the spline order.  ip: penal as a whole number from 0 to 8, or -1.
template <int MODE, int K>
__global__ void __launch_bounds__(ROW_MAX) k_spline_chunks(LevelDims d, const uint8_t* __restrict__ eactive,
                                                           SplineDev sp, const float2* __restrict__ coeff, int ych,
                                                           int cap_j, double rho_min, double penal,
                                                           int ip, double* __restrict__ rho, double* __restrict__ rhop,
                                                           float* __restrict__ rhop32, double* partial, double* out,
                                                           unsigned* ctr, OcStep st) {
  extern __shared__ float2 sC[];  // [cap_j][nb0], then B: [ych][nb0]
  const int nbx = sp.nb[0], nby = sp.nb[1], ex = d.ex;
  float2* sB = sC + (size_t)nbx * cap_j;
  const int x = threadIdx.x, lane = threadIdx.x & 31;
  const bool col = x < ex;
  int ix = -1;
  df nx[K];
#pragma unroll
  for (int r = 0; r < K; ++r) nx[r] = df(0);
  if (col) {
    ix = sp.i0[0][x];
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const float2 n = sp.Ndf[0][x * K + r];
      nx[r] = df(n.x, n.y);
    }
  }
  const df lo = df_from(rho_min), one(1.f, 0.f), outside = df_from(-0.2);
  df sd(0);
  const int ncy = (d.ey + ych - 1) / ych, nchunk = ncy * d.ez;
  for (int c = blockIdx.x; c < nchunk; c += gridDim.x) {
    const int z = c / ncy, y0 = (c - z * ncy) * ych, ny = min(ych, d.ey - y0);
    const int64_t e0 = x + (int64_t)ex * (y0 + (int64_t)d.ey * z);
    unsigned act = 0;  // the column's activity flags, a bit per row
    if (col) {
#pragma unroll
      for (int r = 0; r < CHUNK_Y; ++r)  // all in flight together
        if (r < ny) act |= (eactive[e0 + (int64_t)ex * r] ? 1u : 0u) << r;
    }
    const int iz = sp.i0[2][z];
    // lane r holds row r's first y-basis index (every warp the same)
    const int iy = lane < ny ? sp.i0[1][y0 + lane] : -1;
    const int jlo = __reduce_min_sync(0xffffffffu, iy >= 0 ? iy : nby);
    const int nj = __reduce_max_sync(0xffffffffu, iy >= 0 ? iy + K : jlo) - jlo;
    df nz[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
      const float2 n = sp.Ndf[2][z * K + t];
      nz[t] = df(n.x, n.y);
    }
    __syncthreads();  // the previous chunk's readers are done
    if (iz >= 0 && nj > cap_j) {  // (uniform over the CTA)
      for (int q = threadIdx.x; q < nbx * ny; q += blockDim.x) {
        const df v = spline_yz_at<K>(d, sp, coeff, q % nbx, y0 + q / nbx, iz, nz);
        sB[q] = make_float2(v.hi, v.lo);
      }
    } else if (iz >= 0) {
      for (int q = threadIdx.x; q < nbx * nj; q += blockDim.x) {
        const int j = q / nbx, i = q - j * nbx;
        const float2* cq = coeff + i + (int64_t)nbx * (jlo + j + (int64_t)nby * iz);
        df a(0);
#pragma unroll
        for (int t = 0; t < K; ++t) {
          const float2 cf = cq[(int64_t)nbx * nby * t];
          a += df(cf.x, cf.y) * nz[t];
        }
        sC[q] = make_float2(a.hi, a.lo);
      }
      __syncthreads();
      for (int q = threadIdx.x; q < nbx * ny; q += blockDim.x) {
        const int r = q / nbx, i = q - r * nbx, y = y0 + r;
        const int iyr = sp.i0[1][y];
        df v(0);
        if (iyr >= 0) {
#pragma unroll
          for (int s2 = 0; s2 < K; ++s2) {
            const float2 ns = sp.Ndf[1][y * K + s2];
            const float2 a = sC[i + nbx * (iyr - jlo + s2)];
            v += df(ns.x, ns.y) * df(a.x, a.y);
          }
        }
        sB[q] = make_float2(v.hi, v.lo);
      }
    }
    __syncthreads();
    for (int r0 = 0; r0 < ny; r0 += 4) {  // uniform: every lane takes part in the shuffles
      df v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = r0 + q;
        const int iyr = __shfl_sync(0xffffffffu, iy, r);  // (r < CHUNK_Y; -1 past the chunk)
        const bool in = ix >= 0 && iz >= 0 && iyr >= 0;
        v[q] = in ? df(0) : outside;
        if (in) {
          const float2* b = sB + nbx * r + ix;
#pragma unroll
          for (int t = 0; t < K; ++t) {
            const float2 bb = b[t];
            v[q] += nx[t] * df(bb.x, bb.y);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = r0 + q;
        if (MODE == 0) {
          if (!((act >> r) & 1u)) continue;
          if (df_lt(v[q], lo)) v[q] = lo;
          if (df_lt(one, v[q])) v[q] = one;
          sd += v[q];
        } else {
          if (!col || r >= ny) continue;
          const int64_t e = e0 + (int64_t)ex * r;
          const bool on = (act >> r) & 1u;
          // clamped before the conversion: FP64 compares run on the same pipe as
          // the conversion and the power, which bound this mode (a NaN is rho_min)
          const double vr = !on ? 0.0 : !df_lt(lo, v[q]) ? rho_min : df_lt(v[q], one) ? df_to(v[q]) : 1.0;
          double vp = 0.0;
          if (on) {
            if (ip >= 0) {
              vp = ip > 0 ? vr : 1.0;
              for (int p = 1; p < ip; ++p) vp *= vr;
            } else {
              vp = pow(vr, penal);
            }
          }
          rho[e] = vr; rhop[e] = vp; rhop32[e] = (float)vp;
        }
      }
    }
  }
  if (MODE == 0) finish_volume(df_to(sd), partial, out, ctr, st);
}

// Rows of at most ROW_MAX elements and orders up to MAX_ORDER whose tables fit
// in shared memory go to k_spline_chunks (returns false otherwise).  Chunks of
// CHUNK_Y rows share the z contraction best; a grid with fewer than CHUNK_CTAS
// of them takes shorter ones down to one row, but no more than CHUNK_CTAS (61x37x29
// in 1,073 chunks of a row 715 us an OC update, in 551 of two 631), and tables
// of more than 96 KB (two CTAs on an SM) shorten them too.  A layer's rows are
// dealt evenly to its chunks.
template <int MODE>
static bool spline_chunks(cudaStream_t s, const LevelDims& d, const uint8_t* eactive, const SplineDev& sp,
                          const float2* coeff_df, double rho_min, double penal, double* rho, double* rhop,
                          float* rhop32, double* partial, double* out, unsigned* ctr, const OcStep& st) {
  if (d.ex > ROW_MAX || sp.order < 2 || sp.order > MAX_ORDER) return false;
  int ych = (int)std::min<int64_t>(CHUNK_Y, ((int64_t)d.ey * d.ez + CHUNK_CTAS - 1) / CHUNK_CTAS);
  auto cap = [&](int r) { return std::min(sp.nb[1], r + sp.order - 1); };
  auto bytes = [&](int r) { return sizeof(float2) * (size_t)sp.nb[0] * (cap(r) + r); };
  while (ych > 1 && bytes(ych) > 96 * 1024) --ych;
  const int ncy = (d.ey + ych - 1) / ych;
  ych = (d.ey + ncy - 1) / ncy;
  const size_t smem = bytes(ych);
  if (smem > CHUNK_SMEM) return false;
  auto* fn = sp.order == 2   ? k_spline_chunks<MODE, 2>
             : sp.order == 3 ? k_spline_chunks<MODE, 3>
                             : k_spline_chunks<MODE, 4>;
  // once a device and kernel, for the largest tables: the limit is the kernel's,
  // not the launch's, and designs on other host threads need their own.  Only once
  // tables need it: a raised limit costs the small ones 1 us a launch (191x95x93)
  static PerDeviceOnce once[MAX_ORDER + 1];
  if (smem > 48 * 1024 && once_per_device(once[sp.order], [fn]() -> cudaError_t {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CHUNK_SMEM);
      }) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const int nb = (int)std::min<int64_t>(VOL_BLOCKS, (int64_t)((d.ey + ych - 1) / ych) * d.ez);
  const int ip = penal >= 0.0 && penal <= 8.0 && (double)(int)penal == penal ? (int)penal : -1;
  fn<<<nb, (d.ex + 31) / 32 * 32, smem, s>>>(d, eactive, sp, coeff_df, ych, cap(ych), rho_min, penal, ip, rho, rhop,
                                             rhop32, partial, out, ctr, st);
  return true;
}

void launch_coeff_to_density(cudaStream_t s, const LevelDims& d, const uint8_t* eactive,
                             const SplineDev& sp, const double* coeff, double rho_min, double penal,
                             double* rho, double* rhop, float* rhop32, double* Btmp, float2* coeff_df) {
  const int64_t nB = (int64_t)sp.nb[0] * d.ey * d.ez;
  const int64_t nc = (int64_t)sp.nb[0] * sp.nb[1] * sp.nb[2];
  if (coeff_df) {
    k_to_df<<<nblk(nc, 256), 256, 0, s>>>(nc, coeff, coeff_df);
    if (spline_chunks<1>(s, d, eactive, sp, coeff_df, rho_min, penal, rho, rhop, rhop32, nullptr, nullptr, nullptr,
                         OcStep{}))
      return;
  }
  float2* B = reinterpret_cast<float2*>(Btmp);  // nB (hi, lo) pairs in the nB-double scratch
  k_spline_yz<<<nblk(nB, 256), 256, 0, s>>>(d, sp, coeff, B);
  k_density_from_B<<<nblk(d.ne, 256), 256, 0, s>>>(d, eactive, sp, B, rho_min, penal, rho, rhop, rhop32);
}

int launch_trial_volume(cudaStream_t s, const LevelDims& d, const uint8_t* eactive,
                        const SplineDev& sp, const float2* coeff_df, double rho_min, double* partial,
                        double* out, double* Btmp, unsigned* ctr, OcStep st) {
  if (spline_chunks<0>(s, d, eactive, sp, coeff_df, rho_min, 0.0, nullptr, nullptr, nullptr, partial, out, ctr, st))
    return 1;
  const int64_t nB = (int64_t)sp.nb[0] * d.ey * d.ez;
  float2* B = reinterpret_cast<float2*>(Btmp);  // nB (hi, lo) pairs in the nB-double scratch
  k_spline_yz_df<<<nblk(nB, 256), 256, 0, s>>>(d, sp, coeff_df, B);
  // two elements per thread at most
  const int nb = (int)std::min<int64_t>(VOL_BLOCKS, (d.ne + VOL_THREADS * 2 - 1) / (VOL_THREADS * 2));
  k_volume_from_B<<<nb < 1 ? 1 : nb, VOL_THREADS, 0, s>>>(d, eactive, sp, B, rho_min, partial, out, ctr, st);
  return 2;
}

// Element sensitivity g_e = -p rho^(p-1) u_e^T Ke u_e (optimization/optimization.cu:96-159),
// with u_e^T Ke u_e in the modal form of the fine operator: the transforms of
// the nodal values are exact, on 64-bit integers (fx.cuh), and the modes enter
// the isotropic energy as double-float numbers on the FP32 pipe (48 bits of the
// element's largest mode).  rhop: take rho^(p-1) as rhop / rho (a design
// iteration, whose operator was built from rhop), else from rho.
// Bound by instructions, about 1,700 an element.  The double-float form spent
// them on its transforms and on FP64 conversions, three FP64 operations a nodal
// value (191x95x93: 413 us, here 99).
struct SensConst {
  float2 e, f, g;  // FxConst as (hi, lo) floats
};

// a mode in units of 2^-60
__device__ __forceinline__ df mode_df(int64_t c) {
  c += 1 << 13;
  const float hi = __int2float_rn((int)(c >> 38)), lo = __int2float_rn((int)((c >> 14) & 0xffffff));
  return df_fast2sum(hi * 0x1p-22f, lo * 0x1p-46f);
}
__device__ __forceinline__ void add_sq(df& s, df v) { s += v * v; }

__global__ void __launch_bounds__(128) k_sensitivity(LevelDims d, const uint8_t* __restrict__ eactive,
                                                     const double* __restrict__ rho, const double* __restrict__ rhop,
                                                     const double* __restrict__ u, double penal, SensConst k,
                                                     double* __restrict__ sens) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.ne) return;
  if (!eactive[e]) { sens[e] = 0.0; return; }
  const int x = (int)(e % d.ex);
  const int64_t t = e / d.ex;
  const int y = (int)(t % d.ey), z = (int)(t / d.ey);
  int64_t c[3][8];
  int E[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    int ei[8];
    E[i] = 0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int64_t v = (x + (a & 1)) + (int64_t)d.vx * ((y + ((a >> 1) & 1)) + (int64_t)d.vy * (z + (a >> 2)));
      c[i][a] = fx_split(u[i * d.nv + v], ei[a]);
      E[i] = max(E[i], ei[a]);
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) c[i][a] = fx_down(c[i][a], E[i] - ei[a]);
  }
  const bool bad = max(max(E[0], E[1]), E[2]) >= 0x7ff;
  const int X = fx_modes(c, E[0], E[1], E[2]);
  df se(0), sf(0), sg(0), s(0);
  // constant part of the gradient (weight 3)
  add_sq(se, mode_df(c[0][1] + c[1][2] + c[2][4]));
  add_sq(s, mode_df(c[0][1])); add_sq(s, mode_df(c[1][2])); add_sq(s, mode_df(c[2][4]));
  sf += s + s;
  add_sq(sf, mode_df(c[0][2] + c[1][1])); add_sq(sf, mode_df(c[0][4] + c[2][1])); add_sq(sf, mode_df(c[1][4] + c[2][2]));
  se = se + se + se;
  // X, Y and Z parts
  add_sq(se, mode_df(c[1][3] + c[2][5])); add_sq(se, mode_df(c[0][3] + c[2][6])); add_sq(se, mode_df(c[0][5] + c[1][6]));
  add_sq(sf, mode_df(c[0][3])); add_sq(sf, mode_df(c[1][3])); add_sq(sf, mode_df(c[0][5]));
  add_sq(sf, mode_df(c[2][5])); add_sq(sf, mode_df(c[1][6])); add_sq(sf, mode_df(c[2][6]));
  sf = sf + sf + sf;
  add_sq(sf, mode_df(c[1][5] + c[2][3])); add_sq(sf, mode_df(c[0][6] + c[2][3])); add_sq(sf, mode_df(c[0][6] + c[1][5]));
  add_sq(sg, mode_df(c[0][7])); add_sq(sg, mode_df(c[1][7])); add_sq(sg, mode_df(c[2][7]));
  const df w = se * df(k.e.x, k.e.y) + sf * df(k.f.x, k.f.y) + sg * df(k.g.x, k.g.y);
  double q = fx_scale(df_to(w), 2 * (X - 1019));  // u_e^T Ke u_e
  if (bad) q = __longlong_as_double(0x7ff8000000000000ll);
  const double r = rho[e];
  if (rhop) sens[e] = r > 0.0 ? -penal * (rhop[e] * q) / r : 0.0;
  else sens[e] = -penal * simp_pow(r, penal - 1.0) * q;
}

void launch_sensitivity(cudaStream_t s, const LevelDims& d, const uint8_t* eactive,
                        const double* rho, const double* rhop, const double* u, double penal, double lam, double mu,
                        double h, double* sens) {
  auto split = [](double v) {
    const float hi = (float)v;
    return make_float2(hi, (float)(v - (double)hi));
  };
  const SensConst k{split(lam * h / 48.0), split(mu * h / 48.0), split((lam + 4.0 * mu) * h / 144.0)};
  k_sensitivity<<<nblk(d.ne, 128), 128, 0, s>>>(d, eactive, rho, rhop, u, penal, k, sens);
}

// Sensitivity filter (grid/Grid.cu:4130-4229): normalised average over the ball
// r^2 <= R^2, R_int = floor(R + 0.5), weight 1 - 6s^2 + 8s^3 - 3s^4 with s = r/R.
// The ball's offsets and weights depend only on R; they come precomputed (in the
// reference's loop order dx, dy, dz) so no square root is taken per neighbour.
// It runs in double-float arithmetic (about 1e-14 relative): the sensitivities
// and weights arrive split into (hi, lo) floats, the weighted sums run on the
// FP32 pipe, and the quotient is a double-float division (FP32 quotient, one
// correction from the double-float remainder; Dekker 1971).  An FP64 form is
// bound by GB300's FP64 pipe (66 FP64 operations per element).
__device__ __forceinline__ df df_div(df a, df b) {
  const float q1 = __fdiv_rn(a.hi, b.hi);
  const df r = a - b * df(q1, 0.f);
  const float q2 = __fdiv_rn(r.hi, b.hi);
  return df_fast2sum(q1, q2);
}

__global__ void k_filter_df(LevelDims d, const uint8_t* __restrict__ eactive, const float2* __restrict__ src,
                            double* __restrict__ dst, const int4* __restrict__ offs,
                            const float2* __restrict__ wts, int noffs) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.ne) return;
  if (!eactive[e]) { dst[e] = 0.0; return; }
  int x, y, z;
  if (d.ne < (int64_t)1 << 31) {  // 32-bit index arithmetic
    const unsigned ee = (unsigned)e, ex = (unsigned)d.ex, t = ee / ex;
    x = (int)(ee - t * ex);
    y = (int)(t % (unsigned)d.ey);
    z = (int)(t / (unsigned)d.ey);
  } else {
    x = (int)(e % d.ex);
    const int64_t t = e / d.ex;
    y = (int)(t % d.ey);
    z = (int)(t / d.ey);
  }
  df ws(0), gs(0);
  for (int k = 0; k < noffs; ++k) {
    const int4 o = offs[k];
    const int nx = x + o.x, ny = y + o.y, nz = z + o.z;
    if (nx < 0 || ny < 0 || nz < 0 || nx >= d.ex || ny >= d.ey || nz >= d.ez) continue;
    const int64_t n = nx + (int64_t)d.ex * (ny + (int64_t)d.ey * nz);
    if (!eactive[n]) continue;
    const float2 wv = wts[k], sv = src[n];
    const df w(wv.x, wv.y);
    gs += w * df(sv.x, sv.y);
    ws += w;
  }
  dst[e] = df_to(df_div(gs, ws));
}

void launch_filter_df(cudaStream_t s, const LevelDims& d, const uint8_t* eactive, double* sens,
                      float2* sens_df, const int4* offs, const float2* wts, int noffs) {
  k_to_df<<<nblk(d.ne, 256), 256, 0, s>>>(d.ne, sens, sens_df);
  k_filter_df<<<nblk(d.ne, 128), 128, 0, s>>>(d, eactive, sens_df, sens, offs, wts, noffs);
}

// Ball offsets within r^2 <= R^2, R_int = floor(R + 0.5), weight
// 1 - 6s^2 + 8s^3 - 3s^4 with s = r/R (grid/Grid.cu:4156-4209, 4226-4229).
void filter_table(double R, std::vector<int4>& offs, std::vector<double>& w) {
  const int Ri = (int)(R + 0.5);
  const double R2 = R * R;
  offs.clear();
  w.clear();
  for (int dx = -Ri; dx <= Ri; ++dx)
    for (int dy = -Ri; dy <= Ri; ++dy)
      for (int dz = -Ri; dz <= Ri; ++dz) {
        const double r2 = (double)(dx * dx + dy * dy + dz * dz);
        if (r2 > R2) continue;
        const double sv = std::sqrt(r2 / R2), s2 = sv * sv;
        w.push_back(1.0 - 6.0 * s2 + 8.0 * s2 * sv - 3.0 * s2 * s2);
        offs.push_back(make_int4(dx, dy, dz, 0));
      }
}

// Spline adjoint (grid/Grid.cu:3671-3724) as a deterministic separable gather:
// T1[i][y][z] = sum_x g Nx, T2[i][j][z] = sum_y T1 Ny, dc[i][j][k] = sum_z T2 Nz.
// Elements outside the spline range (any axis) and inactive elements contribute 0.
__global__ void k_adj_x(LevelDims d, const uint8_t* __restrict__ eactive, SplineDev sp,
                        const double* __restrict__ g, double* __restrict__ T1) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nbx = sp.nb[0];
  if (gid >= (int64_t)nbx * d.ey * d.ez) return;
  const int i = (int)(gid % nbx);
  const int64_t yz = gid / nbx;
  const int y = (int)(yz % d.ey), z = (int)(yz / d.ey);
  double s = 0.0;
  if (sp.i0[1][y] >= 0 && sp.i0[2][z] >= 0) {
    const int k = sp.order;
    for (int x = sp.lo[0][i]; x < sp.hi[0][i]; ++x) {
      const int ix = sp.i0[0][x];
      if (ix < 0) continue;
      const int r = i - ix;
      if (r < 0 || r >= k) continue;
      const int64_t e = x + (int64_t)d.ex * (y + (int64_t)d.ey * z);
      if (!eactive[e]) continue;
      s += g[e] * sp.N[0][x * k + r];
    }
  }
  T1[gid] = s;  // layout [z][y][i]
}

__global__ void k_adj_y(LevelDims d, SplineDev sp, const double* __restrict__ T1, double* __restrict__ T2) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nbx = sp.nb[0], nby = sp.nb[1];
  if (gid >= (int64_t)nbx * nby * d.ez) return;
  const int i = (int)(gid % nbx);
  const int64_t t = gid / nbx;
  const int j = (int)(t % nby), z = (int)(t / nby);
  const int k = sp.order;
  double s = 0.0;
  for (int y = sp.lo[1][j]; y < sp.hi[1][j]; ++y) {
    const int iy = sp.i0[1][y];
    if (iy < 0) continue;
    const int r = j - iy;
    if (r < 0 || r >= k) continue;
    s += T1[i + (int64_t)nbx * (y + (int64_t)d.ey * z)] * sp.N[1][y * k + r];
  }
  T2[gid] = s;  // layout [z][j][i]
}

__global__ void k_adj_z(LevelDims d, SplineDev sp, const double* __restrict__ T2, double* __restrict__ dc) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nbx = sp.nb[0], nby = sp.nb[1], nbz = sp.nb[2];
  if (gid >= (int64_t)nbx * nby * nbz) return;
  const int i = (int)(gid % nbx);
  const int64_t t = gid / nbx;
  const int j = (int)(t % nby), kk = (int)(t / nby);
  const int k = sp.order;
  double s = 0.0;
  for (int z = sp.lo[2][kk]; z < sp.hi[2][kk]; ++z) {
    const int iz = sp.i0[2][z];
    if (iz < 0) continue;
    const int r = kk - iz;
    if (r < 0 || r >= k) continue;
    s += T2[i + (int64_t)nbx * (j + (int64_t)nby * z)] * sp.N[2][z * k + r];
  }
  dc[gid] = s;
}

void launch_spline_adjoint(cudaStream_t s, const LevelDims& d, const uint8_t* eactive,
                           const SplineDev& sp, const double* sens, double* csens, double* tmp1,
                           double* tmp2) {
  const int64_t n1 = (int64_t)sp.nb[0] * d.ey * d.ez;
  const int64_t n2 = (int64_t)sp.nb[0] * sp.nb[1] * d.ez;
  const int64_t n3 = (int64_t)sp.nb[0] * sp.nb[1] * sp.nb[2];
  k_adj_x<<<nblk(n1, 256), 256, 0, s>>>(d, eactive, sp, sens, tmp1);
  k_adj_y<<<nblk(n2, 256), 256, 0, s>>>(d, sp, tmp1, tmp2);
  k_adj_z<<<nblk(n3, 256), 256, 0, s>>>(d, sp, tmp2, csens);
}

__global__ void k_penalise(int64_t ne, const uint8_t* __restrict__ eactive, const double* __restrict__ rho,
                           double penal, double* __restrict__ rhop, float* __restrict__ rhop32) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const double v = eactive[e] ? simp_pow(rho[e], penal) : 0.0;
  rhop[e] = v;
  rhop32[e] = (float)v;
}

void launch_penalise(cudaStream_t s, int64_t ne, const uint8_t* eactive, const double* rho,
                     double penal, double* rhop, float* rhop32) {
  k_penalise<<<nblk(ne, 256), 256, 0, s>>>(ne, eactive, rho, penal, rhop, rhop32);
}

// Reference precision (the reference keeps rho in FP32 and takes rho^p with
// powf, grid/Grid.cu:1739): rho rounded to FP32, rho^p = powf(rho, p) in FP32.
__global__ void k_penalise_ref32(int64_t ne, const uint8_t* __restrict__ eactive, double* __restrict__ rho,
                                 float penal, double* __restrict__ rhop, float* __restrict__ rhop32) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const float r = (float)rho[e];
  rho[e] = (double)r;
  const float v = eactive[e] ? powf(r, penal) : 0.f;
  rhop[e] = (double)v;
  rhop32[e] = v;
}

void launch_penalise_ref32(cudaStream_t s, int64_t ne, const uint8_t* eactive, double* rho, double penal,
                           double* rhop, float* rhop32) {
  k_penalise_ref32<<<nblk(ne, 256), 256, 0, s>>>(ne, eactive, rho, (float)penal, rhop, rhop32);
}

// x[i] rounded to FP32 in place: the arrays the reference stores as float.
__global__ void k_round_f32(int64_t n, double* __restrict__ x) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = (double)(float)x[i];
}

void launch_round_f32(cudaStream_t s, int64_t n, double* x) {
  if (n > 0) k_round_f32<<<nblk(n, 256), 256, 0, s>>>(n, x);
}

// OC trial on the coefficients (optimization/optimization.cu:559-587):
// c' = clamp(clamp(c (max(-dc,0)/thres)^damp, c-step, c+step), cmin, cmax).
// The threshold is thres, or *thres_p when that is given (the device-side
// bisection).  For damp = 1/2 the power is the correctly rounded square root.
__global__ void k_oc_trial(int64_t nc, const double* __restrict__ cold, const double* __restrict__ csens,
                           double thres, const double* __restrict__ thres_p, double damp, double step,
                           double cmin, double cmax, double* __restrict__ cnew, float2* __restrict__ cnew_df) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  if (thres_p) thres = *thres_p;
  double g = csens[i];
  if (g > 0) g = 0;
  g = fabs(g);
  const double co = cold[i];
  const double q = g / thres;
  double cn = co * (damp == 0.5 ? sqrt(q) : pow(q, damp));
  cn = fmin(fmax(cn, co - step), co + step);
  cn = fmin(fmax(cn, cmin), cmax);
  cnew[i] = cn;
  if (cnew_df) {
    const df v = df_from(cn);
    cnew_df[i] = make_float2(v.hi, v.lo);
  }
}

void launch_oc_trial(cudaStream_t s, int64_t nc, const double* cold, const double* csens, double thres,
                     double damp, double step, double cmin, double cmax, double* cnew, float2* cnew_df,
                     const double* thres_p) {
  k_oc_trial<<<nblk(nc, 256), 256, 0, s>>>(nc, cold, csens, thres, thres_p, damp, step, cmin, cmax, cnew,
                                           cnew_df);
}

}  // namespace topo
