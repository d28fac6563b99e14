// Coarse-level kernels: 27-point 3x3-block stencil apply / Gauss-Seidel,
// trilinear transfers, Galerkin coarse operators and the coarsest dense solve.
#include <cooperative_groups.h>

#include <mutex>

#include "df.cuh"
#include "topo_internal.h"

namespace cg = cooperative_groups;

namespace topo {

static inline unsigned nblk(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Coarse levels below this vertex count run the warp-per-vertex stencil kernels.
constexpr int64_t STENCIL_WARP_MAX_NV = 32768;

// Where entry e (0..8) of vertex v's block for neighbour k (0..26) lives:
// base(v) + k ks() + e es().
//  form 0: [27][9][nv], FP64 levels of STENCIL_WARP_MAX_NV vertices and more
//  form 1: the same in tiles, FP32 levels of that size, which the row kernels
//    serve: the 243 x 32 coefficients of each group of 32 vertices lie together,
//    so a warp of consecutive vertices reads one contiguous block instead of 243
//    arrays (243 x 32 values per started group)
//  form 2: [nv][9][27], the smaller levels, where a warp takes one vertex and
//    lane k its neighbour k: nine reads of 27 consecutive values.  In form 0
//    each of the 243 values was a sector of its own, eight times the bytes
//    through L2 (FP32 Chebyshev step on 18,500 vertices 8.5 -> 6.7 us, eight
//    right-hand sides on 4,200 12.2 -> 8.4 us).
struct StIdx {
  int64_t nv;
  int form;
  __device__ __forceinline__ int64_t base(int64_t v) const {
    return form == 1 ? (v >> 5) * (243 * 32) + (v & 31) : form == 2 ? v * 243 : v;
  }
  __device__ __forceinline__ int64_t ks() const { return form == 1 ? 9 * 32 : form == 2 ? 1 : 9 * nv; }
  __device__ __forceinline__ int64_t es() const { return form == 1 ? 32 : form == 2 ? 27 : nv; }
};

template <typename T>
StIdx st_idx(const LevelDims& d) {
  return StIdx{d.nv, d.nv < STENCIL_WARP_MAX_NV ? 2 : sizeof(T) == 4 ? 1 : 0};
}

// ---------------------------------------------------------------------------
// Stencil apply: y_v = sum_d S(v,d) u_{v+d}  (grid/Grid.cu:2126-2224 residual form).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void stencil_row(const LevelDims& d, const T* __restrict__ st, StIdx si,
                                            const T* __restrict__ u, int x, int y, int z, int64_t v,
                                            T o[3]) {
  o[0] = o[1] = o[2] = T(0);
  const int64_t nv = d.nv, ss = si.es(), sk = si.ks();
  const T* sb = st + si.base(v);
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const int nx = x + k % 3 - 1, ny = y + k / 3 % 3 - 1, nz = z + k / 9 - 1;
    if (nx < 0 || ny < 0 || nz < 0 || nx >= d.vx || ny >= d.vy || nz >= d.vz) continue;
    const int64_t n = nx + (int64_t)d.vx * (ny + (int64_t)d.vy * nz);
    const T u0 = u[n], u1 = u[nv + n], u2 = u[2 * nv + n];
    const T* s = sb + k * sk;
    o[0] += s[0] * u0 + s[ss] * u1 + s[2 * ss] * u2;
    o[1] += s[3 * ss] * u0 + s[4 * ss] * u1 + s[5 * ss] * u2;
    o[2] += s[6 * ss] * u0 + s[7 * ss] * u1 + s[8 * ss] * u2;
  }
}


// ---------------------------------------------------------------------------
// Point-block Gauss-Seidel on a stencil level.  A vertex is nine lanes of a
// warp, (row, neighbour z plane): each forms the products of nine neighbours
// side by side, and the row's sum then passes through its three lanes in
// neighbour order, so every sum and quotient is bit for bit the one a thread
// walking the 27 neighbours forms.  A warp takes three vertices.  The thread-per-vertex form
// (k_stencil_gs) waits for 243 products on the FP64 pipe with a colour's 80 to
// 1500 vertices in a handful of CTAs: 51 us a colour on a level of 637 vertices,
// here 5.5 us in the cluster form.
// ---------------------------------------------------------------------------
constexpr int GS_PER_WARP = 3;                        // vertices of a warp (27 of its lanes)
constexpr int GS_WARPS = 8;                           // warps of a CTA
constexpr int GS_PER_CTA = GS_PER_WARP * GS_WARPS;    // vertices of a CTA

struct GsColour {  // vertices x = cx + 2i, y = cy + 2j, z = cz + 2k of a level
  int cx, cy, cz, hx, hy, cnt;
};
__host__ __device__ inline GsColour gs_colour(const LevelDims& d, int colour) {
  GsColour c;
  c.cx = colour & 1;
  c.cy = (colour >> 1) & 1;
  c.cz = colour >> 2;
  c.hx = (d.vx - c.cx + 1) / 2;
  c.hy = (d.vy - c.cy + 1) / 2;
  c.cnt = c.hx * c.hy * ((d.vz - c.cz + 1) / 2);
  return c;
}

// s / d with rc = 1 / d computed ahead of time: the product with the correctly
// rounded reciprocal, corrected by its exact remainder, which gives the
// correctly rounded quotient (Markstein 1990) without a division's latency on
// the critical path.
template <typename T>
__device__ __forceinline__ T div_by(T s, T d, T rc) {
  const T q = s * rc;
  const T e = fma(fma(-q, d, s), rc, q);
  return isfinite(e) ? e : q;
}

// What a lane's share of a vertex update needs besides u.
template <typename T>
struct GsLane {
  T c[27];       // stencil coefficients of (row, z plane): neighbour (y, x) major, component minor
  T S[3], rc, f; // block entries (row, .), 1 / S(row, row), right-hand side of the row
  int v, at;     // the vertex (-1: none) and its neighbour (-1, -1, plane) in the level
  unsigned ok;   // in-plane neighbours inside the level
};

template <typename T>
__device__ __forceinline__ void gs_load(const LevelDims& d, const T* __restrict__ st, StIdx si,
                                        const uint8_t* __restrict__ vmask, const T* __restrict__ f, GsColour g, int t,
                                        int row, int part, GsLane<T>& L) {
  L.v = -1;
  L.ok = 0;
  L.f = L.S[0] = L.S[1] = L.S[2] = T(0);
  L.rc = T(1);
  if (t < 0 || t >= g.cnt) return;
  const int q = t / g.hx, x = g.cx + 2 * (t - q * g.hx), qz = q / g.hy, y = g.cy + 2 * (q - qz * g.hy), z = g.cz + 2 * qz;
  const int v = x + d.vx * (y + d.vy * z);
  if (!(vmask[v] & 8)) return;
  L.v = v;
  const int64_t ss = si.es(), sk = si.ks(), nv = d.nv;
  const T* sb = st + si.base(v);
  const int nz = z + part - 1;
  L.at = (x - 1) + d.vx * ((y - 1) + d.vy * nz);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int nx = x + k % 3 - 1, ny = y + k / 3 - 1;
    const bool ok = nz >= 0 && nz < d.vz && nx >= 0 && ny >= 0 && nx < d.vx && ny < d.vy;
    L.ok |= ok ? 1u << k : 0u;
    const T* s = sb + (9 * part + k) * sk + 3 * row * ss;
#pragma unroll
    for (int j = 0; j < 3; ++j) L.c[3 * k + j] = ok ? s[j * ss] : T(0);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) L.S[j] = sb[13 * sk + (3 * row + j) * ss];
  L.rc = T(1) / (row == 0 ? L.S[0] : row == 1 ? L.S[1] : L.S[2]);
  L.f = f[row * nv + v];
}

// Updates the warp's vertices; every lane of the warp must call it.
template <typename T>
__device__ __forceinline__ void gs_update(const LevelDims& d, T* u, const GsLane<T>& L, int lane, int row, int part,
                                          bool reverse) {
  const int64_t nv = d.nv;
  T t[9], own = T(0);
  if (L.v >= 0) {
    T w[27];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int n = L.at + k % 3 + d.vx * (k / 3);
#pragma unroll
      for (int j = 0; j < 3; ++j) w[3 * k + j] = (L.ok >> k) & 1u ? __ldcg(u + j * nv + n) : T(0);
    }
    own = __ldcg(u + row * nv + L.v);
#pragma unroll
    for (int k = 0; k < 9; ++k)
      t[k] = fma(L.c[3 * k + 2], w[3 * k + 2], fma(L.c[3 * k], w[3 * k], L.c[3 * k + 1] * w[3 * k + 1]));
  }
  const int b9 = lane - 3 * row - part, b3 = lane - part;  // first lane of the vertex, of its row
  T o = T(0);
#pragma unroll
  for (int ph = 0; ph < 3; ++ph) {
    if (ph > 0) {
      const T in = __shfl_sync(0xffffffffu, o, (b3 + ph - 1) & 31);
      if (part == ph) o = in;
    }
    if (part == ph && L.v >= 0) {
#pragma unroll
      for (int k = 0; k < 9; ++k)
        if ((L.ok >> k) & 1u) o += t[k];
    }
  }
  const T r = L.f - __shfl_sync(0xffffffffu, o, (b3 + 2) & 31);
  // du of the rows in turn (0, 1, 2; reverse: 2, 1, 0); a lane's du is its row's
  const T Sd = row == 0 ? L.S[0] : row == 1 ? L.S[1] : L.S[2];
  const int first = reverse ? 2 : 0, last = 2 - first;
  const T df_ = div_by(r, Sd, L.rc);  // right for row `first`
  const T d1 = __shfl_sync(0xffffffffu, df_, (b9 + 3 * first) & 31);
  const T Sf = reverse ? L.S[2] : L.S[0];
  const T dm = div_by(fma(-Sf, d1, r), Sd, L.rc);  // right for row 1
  const T d2 = __shfl_sync(0xffffffffu, dm, (b9 + 3) & 31);
  // the last row subtracts by column: 0, 1 forward, 1, 2 in reverse
  const T rl = reverse ? fma(-Sf, d1, fma(-L.S[1], d2, r)) : fma(-L.S[1], d2, fma(-Sf, d1, r));
  const T dl = div_by(rl, Sd, L.rc);
  const T du = row == first ? df_ : row == last ? dl : dm;
  if (L.v >= 0 && part == 0) __stcg(u + row * nv + L.v, own + du);
}

// One colour, one launch.
template <typename T>
__global__ void __launch_bounds__(32 * GS_WARPS) k_stencil_gs9(LevelDims d, const T* __restrict__ st, StIdx si,
                                                               const uint8_t* __restrict__ vmask, T* u,
                                                               const T* __restrict__ f, int colour, bool reverse) {
  const int lane = threadIdx.x & 31, g = lane / 9, j = lane - 9 * g, row = j / 3, part = j - 3 * row;
  const int t = (blockIdx.x * GS_WARPS + (threadIdx.x >> 5)) * GS_PER_WARP + g;
  GsLane<T> L;
  gs_load<T>(d, st, si, vmask, f, gs_colour(d, colour), g < GS_PER_WARP ? t : -1, row, part, L);
  gs_update<T>(d, u, L, lane, row, part, reverse);
}

// All colours of all sweeps in one launch of one thread-block cluster, a
// cluster barrier between colours: for levels whose colours hold no more
// vertices than the cluster updates at once.  The stencil part of the next
// colour is loaded before the wait, so a colour costs the barrier, the
// L2 latency of u and the FP64 products of its few vertices.
template <typename T>
__global__ void __launch_bounds__(32 * GS_WARPS) k_stencil_gs_cluster(LevelDims d, const T* __restrict__ st, StIdx si,
                                                                      const uint8_t* __restrict__ vmask, T* u,
                                                                      const T* __restrict__ f, int sweeps,
                                                                      bool reverse) {
  const int lane = threadIdx.x & 31, g = lane / 9, j = lane - 9 * g, row = j / 3, part = j - 3 * row;
  // consecutive groups of three vertices go to different CTAs (SMs)
  const int t = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * GS_PER_WARP + g;
  for (int k = 0; k < 8 * sweeps; ++k) {
    GsLane<T> L;
    gs_load<T>(d, st, si, vmask, f, gs_colour(d, reverse ? 7 - (k & 7) : (k & 7)), g < GS_PER_WARP ? t : -1, row, part,
               L);
    if (k > 0) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    gs_update<T>(d, u, L, lane, row, part, reverse);
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// Thread per vertex: every lane of a warp carries products, which pays where a
// colour has enough vertices to fill the chip by itself (GS_THREAD_MIN).
template <typename T>
__global__ void k_stencil_gs(LevelDims d, const T* __restrict__ st, StIdx si, const uint8_t* __restrict__ vmask,
                             T* u, const T* __restrict__ f, int cx, int cy, int cz, int hx, int hy,
                             int64_t cnt, bool reverse) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= cnt) return;
  const int x = cx + 2 * (int)(t % hx);
  const int64_t t2 = t / hx;
  const int y = cy + 2 * (int)(t2 % hy), z = cz + 2 * (int)(t2 / hy);
  const int64_t v = x + (int64_t)d.vx * (y + (int64_t)d.vy * z);
  if (!(vmask[v] & 8)) return;
  T o[3], S[9], r[3];
  stencil_row<T>(d, st, si, u, x, y, z, v, o);
#pragma unroll
  for (int k = 0; k < 9; ++k) S[k] = st[si.base(v) + 13 * si.ks() + k * si.es()];
#pragma unroll
  for (int c = 0; c < 3; ++c) r[c] = f[c * d.nv + v] - o[c];
  T du[3] = {T(0), T(0), T(0)};
  if (!reverse) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      T s = r[i];
#pragma unroll
      for (int j = 0; j < i; ++j) s -= S[3 * i + j] * du[j];
      du[i] = s / S[4 * i];
    }
  } else {
#pragma unroll
    for (int i = 2; i >= 0; --i) {
      T s = r[i];
#pragma unroll
      for (int j = i + 1; j < 3; ++j) s -= S[3 * i + j] * du[j];
      du[i] = s / S[4 * i];
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) u[i * d.nv + v] += du[i];
}

template <typename T>
__global__ void k_stencil_diag_inv(LevelDims d, const T* __restrict__ st, StIdx si,
                                   const uint8_t* __restrict__ vmask, T* __restrict__ dinv) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= d.nv) return;
  T S[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) S[k] = st[si.base(v) + 13 * si.ks() + k * si.es()];
  const T a = S[0], b = S[1], c = S[2], dd = S[4], e = S[5], f = S[8];
  const T A0 = dd * f - e * e, A1 = c * e - b * f, A2 = b * e - c * dd;
  const T det = a * A0 + b * A1 + c * A2;
  const T inv[9] = {A0, A1, A2, A1, a * f - c * c, b * c - a * e, A2, b * c - a * e, a * dd - b * b};
  const T rd = T(1) / det;
  const bool act = (vmask[v] & 8) != 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) dinv[k * d.nv + v] = act ? inv[k] * rd : T(0);
}

// Row-split stencil kernels: a CTA of 3 x SV threads covers SV vertices, one
// thread per (vertex, row); the three rows of a vertex share its neighbours'
// values through L1.  Three times the threads of a vertex-per-thread kernel keep
// enough loads in flight on the small coarse levels.
constexpr int SV = 64;

template <typename T>
__device__ __forceinline__ T stencil_row_i(const LevelDims& d, const T* __restrict__ st, StIdx si,
                                           const T* __restrict__ u, int x, int y, int z, int64_t v, int row) {
  T o = T(0);
  const int64_t nv = d.nv, ss = si.es(), sk = si.ks();
  const T* sb = st + si.base(v) + 3 * row * ss;
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const int nx = x + k % 3 - 1, ny = y + k / 3 % 3 - 1, nz = z + k / 9 - 1;
    if (nx < 0 || ny < 0 || nz < 0 || nx >= d.vx || ny >= d.vy || nz >= d.vz) continue;
    const int64_t n = nx + (int64_t)d.vx * (ny + (int64_t)d.vy * nz);
    const T* s = sb + k * sk;
    o += s[0] * u[n] + s[ss] * u[nv + n] + s[2 * ss] * u[2 * nv + n];
  }
  return o;
}

template <typename T>
__global__ void __launch_bounds__(3 * SV) k_stencil_apply3(LevelDims d, const T* __restrict__ st, StIdx si,
                                                           const T* __restrict__ u, const T* __restrict__ f,
                                                           T* __restrict__ out, bool residual) {
  const int64_t bo = (int64_t)blockIdx.y * 3 * d.nv;  // right-hand side of the batch
  u += bo;
  if (f) f += bo;
  out += bo;
  const int row = threadIdx.x / SV;
  const int64_t v = (int64_t)blockIdx.x * SV + threadIdx.x % SV;
  if (v >= d.nv) return;
  const int x = (int)(v % d.vx);
  const int64_t t = v / d.vx;
  const int y = (int)(t % d.vy), z = (int)(t / d.vy);
  const T o = stencil_row_i<T>(d, st, si, u, x, y, z, v, row);
  const int64_t i = row * d.nv + v;
  out[i] = residual ? f[i] - o : o;
}

// One Chebyshev step on a stencil level: uout = u + d, d = c_old d + c_new Dinv (f - A u).
template <typename T>
__global__ void __launch_bounds__(3 * SV) k_stencil_cheb(LevelDims d, const T* __restrict__ st, StIdx si,
                                                         const T* __restrict__ u, const T* __restrict__ f,
                                                         T* __restrict__ uout, const T* __restrict__ dinv,
                                                         T* __restrict__ dv, const double* __restrict__ coef,
                                                         bool first) {
  __shared__ T sr[3][SV];
  const int64_t bo = (int64_t)blockIdx.y * 3 * d.nv;  // right-hand side of the batch
  u += bo;
  f += bo;
  uout += bo;
  dv += bo;
  const int row = threadIdx.x / SV, lv = threadIdx.x % SV;
  const int64_t v = (int64_t)blockIdx.x * SV + lv;
  const int64_t nv = d.nv;
  const bool ok = v < nv;
  if (ok) {
    const int x = (int)(v % d.vx);
    const int64_t t = v / d.vx;
    const int y = (int)(t % d.vy), z = (int)(t / d.vy);
    sr[row][lv] = f[row * nv + v] - stencil_row_i<T>(d, st, si, u, x, y, z, v, row);
  }
  __syncthreads();
  if (!ok) return;
  const T zz = dinv[(3 * row) * nv + v] * sr[0][lv] + dinv[(3 * row + 1) * nv + v] * sr[1][lv] +
               dinv[(3 * row + 2) * nv + v] * sr[2][lv];
  const int64_t i = row * nv + v;
  const T c_old = (T)__ldg(coef), c_new = (T)__ldg(coef + 1);
  const T dn = first ? c_new * zz : c_old * dv[i] + c_new * zz;
  dv[i] = dn;
  uout[i] = u[i] + dn;
}

// Warp-per-vertex forms for the small coarse levels, whose row-per-thread
// kernels are latency-bound (a thread walks 27 neighbours in sequence while
// only a few warps per SM are resident): lane k < 27 takes neighbour k, forms
// its three row contributions from 9 stencil and 3 vector loads, and the warp
// sums them with shuffles.  One round of independent loads per vertex.  Small
// levels' stencils stay in L2, so the lanes' scattered stencil reads are cheap.
constexpr int WV = 8;  // vertices (warps) per 256-thread CTA

template <typename T>
__device__ __forceinline__ void stencil_warp_rows(const LevelDims& d, const T* __restrict__ st,
                                                  const T* __restrict__ u, int64_t v, int lane, T o[3]) {
  const int iv = (int)v, t = iv / d.vx, x = iv - t * d.vx, z = t / d.vy, y = t - z * d.vy;
  o[0] = o[1] = o[2] = T(0);
  if (lane < 27) {
    const int kz = lane / 9, ky = (lane - 9 * kz) / 3, kx = lane - 9 * kz - 3 * ky;
    const int nx = x + kx - 1, ny = y + ky - 1, nz = z + kz - 1;
    if (nx >= 0 && ny >= 0 && nz >= 0 && nx < d.vx && ny < d.vy && nz < d.vz) {
      const int n = nx + d.vx * (ny + d.vy * nz), nv = (int)d.nv;
      const T u0 = u[n], u1 = u[nv + n], u2 = u[2 * nv + n];
      const T* sk = st + (int64_t)iv * 243 + lane;  // form 2 (StIdx)
#pragma unroll
      for (int row = 0; row < 3; ++row)
        o[row] = sk[27 * (3 * row)] * u0 + sk[27 * (3 * row + 1)] * u1 + sk[27 * (3 * row + 2)] * u2;
    }
  }
#pragma unroll
  for (int row = 0; row < 3; ++row)
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) o[row] += __shfl_xor_sync(0xffffffffu, o[row], m);
}

template <typename T>
__global__ void __launch_bounds__(32 * WV) k_stencil_apply_warp(LevelDims d, const T* __restrict__ st,
                                                                const T* __restrict__ u, const T* __restrict__ f,
                                                                T* __restrict__ out, bool residual) {
  const int64_t bo = (int64_t)blockIdx.y * 3 * d.nv;  // right-hand side of the batch
  u += bo;
  if (f) f += bo;
  out += bo;
  const int lane = threadIdx.x & 31;
  const int64_t v = (int64_t)blockIdx.x * WV + (threadIdx.x >> 5);
  if (v >= d.nv) return;  // whole warp
  T o[3];
  stencil_warp_rows<T>(d, st, u, v, lane, o);
  if (lane < 3) {
    const int64_t i = lane * d.nv + v;
    const T ol = lane == 0 ? o[0] : (lane == 1 ? o[1] : o[2]);
    out[i] = residual ? f[i] - ol : ol;
  }
}

template <typename T>
__global__ void __launch_bounds__(32 * WV) k_stencil_cheb_warp(LevelDims d, const T* __restrict__ st,
                                                               const T* __restrict__ u, const T* __restrict__ f,
                                                               T* __restrict__ uout, const T* __restrict__ dinv,
                                                               T* __restrict__ dv, const double* __restrict__ coef,
                                                               bool first) {
  const int64_t bo = (int64_t)blockIdx.y * 3 * d.nv;  // right-hand side of the batch
  u += bo;
  f += bo;
  uout += bo;
  dv += bo;
  const int lane = threadIdx.x & 31;
  const int64_t v = (int64_t)blockIdx.x * WV + (threadIdx.x >> 5);
  if (v >= d.nv) return;  // whole warp
  T o[3];
  stencil_warp_rows<T>(d, st, u, v, lane, o);
  if (lane < 3) {
    const int64_t nv = d.nv;
    const T r0 = f[v] - o[0], r1 = f[nv + v] - o[1], r2 = f[2 * nv + v] - o[2];
    const T zz = dinv[(3 * lane) * nv + v] * r0 + dinv[(3 * lane + 1) * nv + v] * r1 +
                 dinv[(3 * lane + 2) * nv + v] * r2;
    const int64_t i = lane * nv + v;
    const T c_old = (T)__ldg(coef), c_new = (T)__ldg(coef + 1);
    const T dn = first ? c_new * zz : c_old * dv[i] + c_new * zz;
    dv[i] = dn;
    uout[i] = u[i] + dn;
  }
}

// The FP64 step on the small levels, nine lanes a vertex as in gs_load: the warp
// form above spends a warp's FP64 issue (16 clocks) on every one of its 15
// shuffle additions and leaves a sixth of its lanes idle; here three vertices
// share a warp and a row is finished by two additions (9,537 and 1,377
// vertices, mean: 16.0 -> 11.2 us).
__global__ void __launch_bounds__(32 * GS_WARPS) k_stencil_cheb9(LevelDims d, const double* __restrict__ st, StIdx si,
                                                                 const double* __restrict__ u,
                                                                 const double* __restrict__ f,
                                                                 double* __restrict__ uout,
                                                                 const double* __restrict__ dinv,
                                                                 double* __restrict__ dv,
                                                                 const double* __restrict__ coef, bool first) {
  const int64_t bo = (int64_t)blockIdx.y * 3 * d.nv;  // right-hand side of the batch
  u += bo;
  f += bo;
  uout += bo;
  dv += bo;
  const int lane = threadIdx.x & 31, g = lane / 9, j9 = lane - 9 * g, row = j9 / 3, part = j9 - 3 * row;
  const int nv = (int)d.nv, v = (blockIdx.x * GS_WARPS + (threadIdx.x >> 5)) * GS_PER_WARP + g;
  const bool ok = g < GS_PER_WARP && v < nv;
  double a[3] = {0.0, 0.0, 0.0}, fr = 0.0, un = 0.0, dn = 0.0, di[3] = {0.0, 0.0, 0.0};
  const int i = row * nv + v;
  if (ok) {
    fr = f[i];
    un = u[i];
    dn = first ? 0.0 : dv[i];
#pragma unroll
    for (int c = 0; c < 3; ++c) di[c] = dinv[(3 * row + c) * (int64_t)nv + v];
    const int t = v / d.vx, x = v - t * d.vx, z = t / d.vy, y = t - z * d.vy, nz = z + part - 1;
    const int64_t es = si.es(), ks = si.ks();
    const double* sb = st + si.base(v) + 3 * row * es + 9 * part * ks;
    if (nz >= 0 && nz < d.vz) {
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const int nx = x + k % 3 - 1, ny = y + k / 3 - 1;
        if (nx < 0 || ny < 0 || nx >= d.vx || ny >= d.vy) continue;
        const int n = nx + d.vx * (ny + d.vy * nz);
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] += sb[k * ks + c * es] * u[c * nv + n];
      }
    }
  }
  const double s = (a[0] + a[1]) + a[2];
  const int b9 = lane - j9, b3 = lane - part;
  const double r = fr - ((__shfl_sync(0xffffffffu, s, b3 & 31) + __shfl_sync(0xffffffffu, s, (b3 + 1) & 31)) +
                         __shfl_sync(0xffffffffu, s, (b3 + 2) & 31));
  const double r0 = __shfl_sync(0xffffffffu, r, b9 & 31), r1 = __shfl_sync(0xffffffffu, r, (b9 + 3) & 31),
               r2 = __shfl_sync(0xffffffffu, r, (b9 + 6) & 31);
  if (!ok || part) return;
  const double z = di[0] * r0 + di[1] * r1 + di[2] * r2, c_old = __ldg(coef), c_new = __ldg(coef + 1);
  dn = first ? c_new * z : c_old * dn + c_new * z;
  dv[i] = dn;
  uout[i] = un + dn;
}

// Levels with fewer vertices than this use the warp-per-vertex kernels.

template <typename T>
void launch_stencil_apply(cudaStream_t s, const LevelDims& d, const T* st, const T* u, const T* f,
                          T* out, bool residual, int nb) {
  if (d.nv < STENCIL_WARP_MAX_NV)
    k_stencil_apply_warp<T><<<dim3(nblk(d.nv, WV), nb), 32 * WV, 0, s>>>(d, st, u, f, out, residual);
  else
    k_stencil_apply3<T><<<dim3(nblk(d.nv, SV), nb), 3 * SV, 0, s>>>(d, st, st_idx<T>(d), u, f, out, residual);
}

template <typename T>
void launch_stencil_cheb(cudaStream_t s, const LevelDims& d, const T* st, const T* u, const T* f, T* uout,
                         const T* dinv, T* dvec, const double* coef, bool first, int nb) {
  if constexpr (sizeof(T) == 8) {
    if (d.nv < STENCIL_WARP_MAX_NV) {
      k_stencil_cheb9<<<dim3(nblk(d.nv, GS_PER_CTA), nb), 32 * GS_WARPS, 0, s>>>(d, st, st_idx<T>(d), u, f, uout, dinv,
                                                                                dvec, coef, first);
      return;
    }
  } else if (d.nv < STENCIL_WARP_MAX_NV) {
    k_stencil_cheb_warp<T><<<dim3(nblk(d.nv, WV), nb), 32 * WV, 0, s>>>(d, st, u, f, uout, dinv, dvec, coef, first);
    return;
  }
  k_stencil_cheb<T><<<dim3(nblk(d.nv, SV), nb), 3 * SV, 0, s>>>(d, st, st_idx<T>(d), u, f, uout, dinv, dvec, coef,
                                                                first);
}

template void launch_stencil_cheb<double>(cudaStream_t, const LevelDims&, const double*, const double*,
                                          const double*, double*, const double*, double*, const double*, bool, int);
template void launch_stencil_cheb<float>(cudaStream_t, const LevelDims&, const float*, const float*,
                                         const float*, float*, const float*, float*, const double*, bool, int);

// First Chebyshev step from a zero iterate with a stored block-Jacobi inverse
// (coarse levels; FP64 level 0 with its free-DOF mask): r = f, d = c_new D^-1 r,
// u_out = d.  Equals the full step on u = 0, since A 0 = 0 exactly.
template <typename T>
__global__ void k_cheb_zero_stored(int64_t nv, const uint8_t* __restrict__ vmask, const T* __restrict__ dinv,
                                   const T* __restrict__ f, T* __restrict__ dv, T* __restrict__ uout,
                                   const double* __restrict__ coef) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const int64_t bo = (int64_t)blockIdx.y * 3 * nv;
  f += bo;
  dv += bo;
  uout += bo;
  const uint8_t m = vmask ? vmask[v] : 7;
  T r[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) r[c] = ((m >> c) & 1) ? f[c * nv + v] : T(0);
  const T c_new = (T)__ldg(coef + 1);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T zz = dinv[(3 * c) * nv + v] * r[0] + dinv[(3 * c + 1) * nv + v] * r[1] + dinv[(3 * c + 2) * nv + v] * r[2];
    const T dn = c_new * zz;
    dv[c * nv + v] = dn;
    uout[c * nv + v] = dn;
  }
}

template <typename T>
void launch_cheb_zero_stored(cudaStream_t s, int64_t nv, const uint8_t* vmask, const T* dinv, const T* f, T* dvec,
                             T* uout, const double* coef, int nb) {
  k_cheb_zero_stored<T><<<dim3(nblk(nv, 256), nb), 256, 0, s>>>(nv, vmask, dinv, f, dvec, uout, coef);
}

template void launch_cheb_zero_stored<double>(cudaStream_t, int64_t, const uint8_t*, const double*, const double*,
                                              double*, double*, const double*, int);
template void launch_cheb_zero_stored<float>(cudaStream_t, int64_t, const uint8_t*, const float*, const float*,
                                             float*, float*, const double*, int);

// CTAs of the cluster k_stencil_gs_cluster runs in: 16 where the device can
// place such a cluster (more SMs share the FP64 work of a colour), else 8.
template <typename T>
static int gs_cluster_size() {
  static PerDeviceOnce once;
  static std::atomic<int> size[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 8;
  const cudaError_t e = once_per_device(once, [&]() -> cudaError_t {
    int n = 0;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(16);
    c.blockDim = dim3(32 * GS_WARPS);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 16;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    const bool big = cudaFuncSetAttribute(k_stencil_gs_cluster<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                         cudaSuccess &&
                     cudaOccupancyMaxActiveClusters(&n, k_stencil_gs_cluster<T>, &c) == cudaSuccess && n > 0;
    cudaGetLastError();
    size[dev] = big ? 16 : 8;
    return cudaSuccess;
  });
  return e == cudaSuccess ? size[dev].load() : 8;
}

// A colour of at least this many vertices runs thread per vertex.  Us a colour,
// nine lanes against one thread a vertex, FP64: 400 vertices 10.4 / 24.7, 1,200
// 12.2 / 24.7, 8,800 29.5 / 45.8, 20,000 58.4 / 53.6, 29,000 83 / 57; FP32: 1,200
// 4.8 / 18, 8,800 8.6 / 23, 17,000 13.7 / 24, 29,000 20.4 / 25, 43,500 29 / 28,
// 56,000 38 / 32.
template <typename T>
constexpr int GS_THREAD_MIN = sizeof(T) == 8 ? 16384 : 40960;

// `sweeps` Gauss-Seidel sweeps, colours 0..7 or 7..0.  Returns the launches made.
template <typename T>
int launch_stencil_gs(cudaStream_t s, const LevelDims& d, const T* st, const uint8_t* vmask, T* u,
                      const T* f, int sweeps, bool reverse) {
  if (sweeps <= 0 || d.nv <= 0) return 0;
  const GsColour big = gs_colour(d, 0);  // the largest colour
  const int cl = gs_cluster_size<T>();
  if (big.cnt <= cl * GS_PER_CTA) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(cl);
    c.blockDim = dim3(32 * GS_WARPS);
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cl;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, k_stencil_gs_cluster<T>, d, st, st_idx<T>(d), vmask, u, f, sweeps, reverse);
    return 1;
  }
  int n = 0;
  for (int sw = 0; sw < sweeps; ++sw)
    for (int cc = 0; cc < 8; ++cc) {
      const int col = reverse ? 7 - cc : cc;
      const GsColour g = gs_colour(d, col);
      if (g.cnt <= 0) continue;
      if (big.cnt >= GS_THREAD_MIN<T>)
        k_stencil_gs<T><<<nblk(g.cnt, 128), 128, 0, s>>>(d, st, st_idx<T>(d), vmask, u, f, g.cx, g.cy, g.cz, g.hx, g.hy,
                                                       g.cnt, reverse);
      else
        k_stencil_gs9<T><<<nblk(g.cnt, GS_PER_CTA), 32 * GS_WARPS, 0, s>>>(d, st, st_idx<T>(d), vmask, u, f, col,
                                                                          reverse);
      ++n;
    }
  return n;
}

template <typename T>
void launch_stencil_diag_inv(cudaStream_t s, const LevelDims& d, const T* st, const uint8_t* vmask,
                             T* dinv) {
  k_stencil_diag_inv<T><<<nblk(d.nv, 256), 256, 0, s>>>(d, st, st_idx<T>(d), vmask, dinv);
}

// ---------------------------------------------------------------------------
// Transfers.  Prolongation is trilinear interpolation from the coarse element
// corners, masked on fixed fine DOFs; restriction is its exact transpose
// (factor 4: grid/Grid.cu:2509-2570 and 2635-2671; factor 2: 2456-2507, 2594-2632).
// ---------------------------------------------------------------------------
template <typename T, int FCT>
__global__ void k_restrict(LevelDims fd, LevelDims cd, const T* __restrict__ rf, T* __restrict__ fc) {
  rf += (int64_t)blockIdx.y * 3 * fd.nv;  // right-hand side of the batch
  fc += (int64_t)blockIdx.y * 3 * cd.nv;
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= cd.nv) return;
  const int x = (int)(v % cd.vx);
  const int64_t t = v / cd.vx;
  const int y = (int)(t % cd.vy), z = (int)(t / cd.vy);
  T s0 = T(0), s1 = T(0), s2 = T(0);
  const T inv = T(1) / T(FCT * FCT * FCT);
  for (int dz = -(FCT - 1); dz <= FCT - 1; ++dz) {
    const int fz = z * FCT + dz;
    if (fz < 0 || fz >= fd.vz) continue;
    const int wz = FCT - (dz < 0 ? -dz : dz);
    for (int dy = -(FCT - 1); dy <= FCT - 1; ++dy) {
      const int fy = y * FCT + dy;
      if (fy < 0 || fy >= fd.vy) continue;
      const int wyz = wz * (FCT - (dy < 0 ? -dy : dy));
#pragma unroll
      for (int dx = -(FCT - 1); dx <= FCT - 1; ++dx) {
        const int fx = x * FCT + dx;
        if (fx < 0 || fx >= fd.vx) continue;
        const T w = T(wyz * (FCT - (dx < 0 ? -dx : dx))) * inv;
        const int64_t fv = fx + (int64_t)fd.vx * (fy + (int64_t)fd.vy * fz);
        s0 += w * rf[fv];
        s1 += w * rf[fd.nv + fv];
        s2 += w * rf[2 * fd.nv + fv];
      }
    }
  }
  fc[v] = s0; fc[cd.nv + v] = s1; fc[2 * cd.nv + v] = s2;
}

// Restriction by a factor of 4 with the fine z taps split across warps: a CTA
// of 7 warps covers 32 consecutive coarse vertices; warp w gathers the fine
// plane z = 4 cz + w - 3 (7 x 7 taps, weights (4 - |d|) per axis) for its lane's
// vertex, and warp 0 sums the seven partial sums in a fixed order.  Seven
// times the threads of a vertex-per-thread gather keep the loads in flight.
constexpr int R4_WARPS = 7;
// FP64 asks for a warp's 49 taps together instead of a row of 7 at a time, which
// waits less at every size (CTAs: us row / all; 20: 18.0 / 14.4, 133 18.5 / 14.4, 299
// 26.7 / 24.5, 566 51.6 / 43.1, 2,213 175 / 147).  FP32 has enough of them in flight
// by the row on the grids that it takes (8 x 133 CTAs: 20 us, all 25), with branches
// past the grid's sides (159x79x77: 13.5 us, with selects 15.5).

template <typename T>
__global__ void __launch_bounds__(32 * R4_WARPS) k_restrict4(LevelDims fd, LevelDims cd, const T* __restrict__ rf,
                                                             T* __restrict__ fc) {
  constexpr bool FLAT = sizeof(T) == 8;
  __shared__ T part[R4_WARPS][3][32];
  rf += (int64_t)blockIdx.y * 3 * fd.nv;  // right-hand side of the batch
  fc += (int64_t)blockIdx.y * 3 * cd.nv;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t v = (int64_t)blockIdx.x * 32 + lane;
  T s0 = T(0), s1 = T(0), s2 = T(0);
  if (v < cd.nv) {
    const int x = (int)(v % cd.vx);
    const int64_t t = v / cd.vx;
    const int y = (int)(t % cd.vy), z = (int)(t / cd.vy);
    const int dz = w - 3, fz = 4 * z + dz;
    if (fz >= 0 && fz < fd.vz) {
      const T wz = T(4 - (dz < 0 ? -dz : dz));
      auto taps = [&](int dy) {
        const int fy = 4 * y + dy;
        const bool iny = fy >= 0 && fy < fd.vy;
        if (!FLAT && !iny) return;
        const T wyz = wz * T(4 - (dy < 0 ? -dy : dy));
        const int64_t rowv = (int64_t)fd.vx * (fy + (int64_t)fd.vy * fz);
#pragma unroll
        for (int dx = -3; dx <= 3; ++dx) {
          const int fx = 4 * x + dx;
          const bool in = iny && fx >= 0 && fx < fd.vx;
          const T wt = wyz * T(4 - (dx < 0 ? -dx : dx));
          const int64_t fv = rowv + fx;
          if constexpr (FLAT) {
            s0 += wt * (in ? rf[fv] : T(0));
            s1 += wt * (in ? rf[fd.nv + fv] : T(0));
            s2 += wt * (in ? rf[2 * fd.nv + fv] : T(0));
          } else if (in) {
            s0 += wt * rf[fv];
            s1 += wt * rf[fd.nv + fv];
            s2 += wt * rf[2 * fd.nv + fv];
          }
        }
      };
      if constexpr (FLAT) {
#pragma unroll
        for (int dy = -3; dy <= 3; ++dy) taps(dy);
      } else {
        for (int dy = -3; dy <= 3; ++dy) taps(dy);
      }
    }
  }
  part[w][0][lane] = s0;
  part[w][1][lane] = s1;
  part[w][2][lane] = s2;
  __syncthreads();
  if (w == 0 && v < cd.nv) {
    const T inv = T(1) / T(64);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T a = T(0);
#pragma unroll
      for (int k = 0; k < R4_WARPS; ++k) a += part[k][c][lane];
      fc[c * cd.nv + v] = a * inv;
    }
  }
}

// The same with a coarse vertex on eight lanes, one x tap each (seven used): a
// lane has 21 taps instead of 147 and a warp's loads are 19 neighbouring values,
// so a grid of a few CTAs becomes eight times as many that each wait once.
template <typename T>
__global__ void __launch_bounds__(32 * R4_WARPS) k_restrict4_lanes(LevelDims fd, LevelDims cd,
                                                                   const T* __restrict__ rf, T* __restrict__ fc) {
  __shared__ T part[R4_WARPS][3][4];
  rf += (int64_t)blockIdx.y * 3 * fd.nv;  // right-hand side of the batch
  fc += (int64_t)blockIdx.y * 3 * cd.nv;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 3, tap = lane & 7;
  const int64_t v0 = (int64_t)blockIdx.x * 4, v = v0 + g;
  T s0 = T(0), s1 = T(0), s2 = T(0);
  if (v < cd.nv && tap < 7) {
    const int t = (int)(v / cd.vx), x = (int)(v - (int64_t)t * cd.vx), z = t / cd.vy, y = t - z * cd.vy;
    const int fx = 4 * x + tap - 3, fz = 4 * z + w - 3;
    if (fx >= 0 && fx < fd.vx && fz >= 0 && fz < fd.vz) {
#pragma unroll
      for (int dy = -3; dy <= 3; ++dy) {
        const int fy = 4 * y + dy;
        const bool in = fy >= 0 && fy < fd.vy;
        const T wy = T(4 - (dy < 0 ? -dy : dy));
        const int64_t fv = in ? fx + (int64_t)fd.vx * (fy + (int64_t)fd.vy * fz) : 0;
        s0 += wy * (in ? rf[fv] : T(0));
        s1 += wy * (in ? rf[fd.nv + fv] : T(0));
        s2 += wy * (in ? rf[2 * fd.nv + fv] : T(0));
      }
      const T wt = T((w < 3 ? w + 1 : 7 - w) * (tap < 3 ? tap + 1 : 7 - tap));
      s0 *= wt;
      s1 *= wt;
      s2 *= wt;
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (tap == 0) {
    part[w][0][g] = s0;
    part[w][1][g] = s1;
    part[w][2][g] = s2;
  }
  __syncthreads();
  if (tid < 12 && v0 + (tid & 3) < cd.nv) {
    const int c = tid >> 2, q = tid & 3;
    T a = T(0);
#pragma unroll
    for (int k = 0; k < R4_WARPS; ++k) a += part[k][c][q];
    fc[c * cd.nv + v0 + q] = a * (T(1) / T(64));
  }
}

template <typename T, int FCT>
__global__ void k_prolong(LevelDims fd, LevelDims cd, const T* __restrict__ uc, T* __restrict__ uf,
                          const uint8_t* __restrict__ vmask) {
  uc += (int64_t)blockIdx.y * 3 * cd.nv;  // right-hand side of the batch
  uf += (int64_t)blockIdx.y * 3 * fd.nv;
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= fd.nv) return;
  int x, y, z;
  if (fd.nv < (int64_t)1 << 31) {  // 32-bit index arithmetic
    const unsigned vv = (unsigned)v, vx = (unsigned)fd.vx, vy = (unsigned)fd.vy, tt = vv / vx;
    x = (int)(vv - tt * vx);
    y = (int)(tt % vy);
    z = (int)(tt / vy);
  } else {
    x = (int)(v % fd.vx);
    const int64_t t = v / fd.vx;
    y = (int)(t % fd.vy);
    z = (int)(t / fd.vy);
  }
  const uint8_t m = vmask[v];
  if (!(m & 7) || !(m & 8)) return;
  const int cx = x / FCT, cy = y / FCT, cz = z / FCT;
  const int rx = x % FCT, ry = y % FCT, rz = z % FCT;
  T s0 = T(0), s1 = T(0), s2 = T(0);
  const T inv = T(1) / T(FCT * FCT * FCT);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ox = k & 1, oy = (k >> 1) & 1, oz = k >> 2;
    const int wx = ox ? rx : FCT - rx, wy = oy ? ry : FCT - ry, wz = oz ? rz : FCT - rz;
    const int wi = wx * wy * wz;
    if (wi == 0) continue;
    const T w = T(wi) * inv;
    const int64_t cv = (cx + ox) + (int64_t)cd.vx * ((cy + oy) + (int64_t)cd.vy * (cz + oz));
    s0 += w * uc[cv];
    s1 += w * uc[cd.nv + cv];
    s2 += w * uc[2 * cd.nv + cv];
  }
  if (m & 1) uf[v] += s0;
  if (m & 2) uf[fd.nv + v] += s1;
  if (m & 4) uf[2 * fd.nv + v] += s2;
}

// Up to three CTAs of the row form per SM the lanes form is the faster one (CTAs
// of the row form, us lanes / row: 20 3.2 / 9.7, 95 4.8 / 10.8, 232 8.1 / 11.7, 299
// 9.0 / 12.8, 354 10.3 / 11.9, 418 11.5 / 12.7, 566 14.5 / 14.3, 1,064 24 / 20, 2,212
// 47 / 43: it reads each fine plane by more CTAs).
// FP32 only: the FP64 forms keep the order of their sums, which callers of
// nearly converged cycles see in the residual's last digits.
constexpr unsigned R4_LANES_CTAS = 456;
template <typename T>
void launch_restrict(cudaStream_t s, const LevelDims& fine, const LevelDims& coarse, const T* rf,
                     T* fc, int nb) {
  if (coarse.factor == 4) {
    const unsigned g = nblk(coarse.nv, 32);
    if constexpr (sizeof(T) == 4) {
      if (g * (unsigned)nb < R4_LANES_CTAS) {
        k_restrict4_lanes<T><<<dim3(nblk(coarse.nv, 4), nb), 32 * R4_WARPS, 0, s>>>(fine, coarse, rf, fc);
        return;
      }
    }
    k_restrict4<T><<<dim3(g, nb), 32 * R4_WARPS, 0, s>>>(fine, coarse, rf, fc);
  } else {
    k_restrict<T, 2><<<dim3(nblk(coarse.nv, 128), nb), 128, 0, s>>>(fine, coarse, rf, fc);
  }
}

// Prolongation by a factor of 4: a warp takes a piece of a row, up to 96 fine
// vertices.  Lane l forms the y-z combination of coarse column cx0 + l once (25 of
// them cover a piece), and a fine vertex takes its two by shuffles; masks, fine
// values and stores are lane by lane along x, whole lines: 103 MB at 256x128x128 in
// 23 us.  (A thread per four neighbouring vertices wrote every fourth value of a
// line at a time, 40 us; 48x24x24 5.2 -> 3.8 us.)
// FP64 is bound by its pipe, 16 clocks of an SM for an instruction of a warp
// whatever its lanes do: there a row's units of 32 vertices are dealt evenly to its
// pieces and no others are worked on (FP32 keeps pieces of 96: dealt, 28 against
// 24 us at 256x128x128), a value and
// component takes two operations, and the weights come from integers without
// conversion.  FP64, us,
// a thread per four vertices / pieces of 96 from the row's start with three
// operations / this: 61x37x29 8.3 / 6.5 / 6.3, 128x64x64 21.7 / 24.8 / 16.8,
// 192x96x96 55.5 / 73.9 / 43.0, 256x128x128 119 / 128 / 82.
constexpr int P4_EACH = 3;  // units of 32 fine vertices of a warp, at most
static_assert(32 * P4_EACH / 4 + 1 <= 32, "a lane per coarse column of a piece");

// w as T, 1 <= w <= 16
template <typename T>
__device__ __forceinline__ T small_weight(int w) {
  const float f = (float)w;
  if constexpr (sizeof(T) == 4) return f;
  else return __hiloint2double((__float_as_int(f) >> 3) + (896 << 20), 0);
}

template <typename T>
__global__ void __launch_bounds__(256) k_prolong4x(LevelDims fd, LevelDims cd, const T* __restrict__ uc,
                                                   T* __restrict__ uf, const uint8_t* __restrict__ vmask, int units,
                                                   int pieces) {
  uc += (int64_t)blockIdx.y * 3 * cd.nv;  // right-hand side of the batch
  uf += (int64_t)blockIdx.y * 3 * fd.nv;
  const int lane = threadIdx.x & 31;
  const int64_t q = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);  // this warp's piece
  const int64_t row = q / pieces;
  if (row >= (int64_t)fd.vy * fd.vz) return;
  const int piece = (int)(q - row * pieces), z = (int)(row / fd.vy), y = (int)(row - (int64_t)z * fd.vy);
  int n = P4_EACH, x0 = 32 * P4_EACH * piece;  // units of this piece and its first vertex
  if constexpr (sizeof(T) == 8) {
    const int uq = units / pieces, ur = units - uq * pieces;
    n = uq + (piece < ur ? 1 : 0);
    x0 = 32 * (piece * uq + min(piece, ur));
  }
  const int64_t v0 = row * fd.vx;
  uint8_t mm[P4_EACH];
  T uo[P4_EACH][3];
#pragma unroll
  for (int k = 0; k < P4_EACH; ++k) {
    const int x = x0 + 32 * k + lane;
    const bool in = (sizeof(T) == 4 || k < n) && x < fd.vx;
    mm[k] = in ? vmask[v0 + x] : 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) uo[k][c] = in ? uf[c * fd.nv + v0 + x] : T(0);
  }
  const int cx = x0 / 4 + lane, cy = y / 4, cz = z / 4, ry = y % 4, rz = z % 4;
  // corners with a zero weight are not read (they may lie outside the coarse grid)
  T cyz[3] = {T(0), T(0), T(0)};  // sum over oy, oz of wy wz u_c
  if (lane <= 8 * (sizeof(T) == 8 ? n : P4_EACH) && cx < cd.vx) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int oy = k & 1, oz = k >> 1;
      const int w = (oy ? ry : 4 - ry) * (oz ? rz : 4 - rz);
      if (w == 0) continue;
      const T wt = small_weight<T>(w);
      const int64_t cv = cx + (int64_t)cd.vx * ((cy + oy) + (int64_t)cd.vy * (cz + oz));
      cyz[0] += wt * uc[cv];
      cyz[1] += wt * uc[cd.nv + cv];
      cyz[2] += wt * uc[2 * cd.nv + cv];
    }
  }
  // ((4 - rx) a + rx b) / 64 with one rounding.  FP64: rx = 0, 2 as a, a + b and 1, 3
  // as 3 a + b, a + 3 b in a fused multiply-add, the power of two with the 1 / 64.
  // FP32: the product by 3, if there is one, in the fused multiply-add, the other
  // weight a power of two or 0 (by the FP64 form 26 against 24 us at 256x128x128).
  const int rx = lane & 3;
  T wm, sc, wq = T(0);
  if constexpr (sizeof(T) == 8) {
    wm = rx & 1 ? T(3) : T(1);
    sc = rx == 0 ? T(1) / T(16) : rx == 2 ? T(1) / T(32) : T(1) / T(64);
  } else {
    wm = T(rx == 3 ? 3 : 4 - rx);
    wq = T(rx == 3 ? 1 : rx);
    sc = T(1) / T(64);
  }
#pragma unroll
  for (int k = 0; k < P4_EACH; ++k) {
    if (sizeof(T) == 8 && k >= n) break;  // the whole warp
    const uint8_t m = (mm[k] & 8) ? mm[k] : 0;
    const int from = 8 * k + (lane >> 2);
    const int64_t v = v0 + x0 + 32 * k + lane;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T a = __shfl_sync(0xffffffffu, cyz[c], from), b = __shfl_sync(0xffffffffu, cyz[c], from + 1);
      T t;
      if constexpr (sizeof(T) == 8) t = fma(wm, rx == 3 ? b : a, rx == 0 ? T(0) : rx == 3 ? a : b);
      else t = fma(wm, rx == 3 ? b : a, wq * (rx == 3 ? a : b));
      if ((m >> c) & 1) uf[c * fd.nv + v] = uo[k][c] + t * sc;
    }
  }
}

template <typename T>
void launch_prolong(cudaStream_t s, const LevelDims& fine, const LevelDims& coarse, const T* uc,
                    T* uf, const uint8_t* vmask_fine, int nb) {
  if (coarse.factor == 4) {
    const int units = (fine.vx + 31) / 32, pieces = (units + P4_EACH - 1) / P4_EACH;
    k_prolong4x<T><<<dim3(nblk((int64_t)pieces * fine.vy * fine.vz, 8), nb), 256, 0, s>>>(fine, coarse, uc, uf,
                                                                                         vmask_fine, units, pieces);
  } else
    k_prolong<T, 2><<<dim3(nblk(fine.nv, 256), nb), 256, 0, s>>>(fine, coarse, uc, uf, vmask_fine);
}

// ---------------------------------------------------------------------------
// Galerkin, first coarse level (grid/Grid.cu:1111-1225 restated per element):
// K_E = sum_pos rho^p_pos T_pos over fine elements without fixed DOFs (a
// [N_E x 64] x [64 x 300] product over the symmetric entries), plus the exact
// Q^T Ktilde Q of fine elements that touch fixed DOFs, where Ktilde has the
// fixed rows/columns zeroed and 1e6 on their diagonal (grid/Grid.cu:1196-1207).
// ---------------------------------------------------------------------------
constexpr int GAL_CE = 16;    // coarse elements per CTA
constexpr int GAL_THREADS = 320;

template <typename T, int FCT>
__global__ void __launch_bounds__(GAL_THREADS) k_galerkin_gemm(LevelDims fd, LevelDims cd,
                                                               const double* __restrict__ rhop,
                                                               const uint8_t* __restrict__ vmask,
                                                               const T* __restrict__ Ttab,
                                                               T* __restrict__ kel) {
  constexpr int NPOS = FCT * FCT * FCT;
  __shared__ T rp[GAL_CE][NPOS];
  const int64_t ce0 = (int64_t)blockIdx.x * GAL_CE;
  for (int i = threadIdx.x; i < GAL_CE * NPOS; i += blockDim.x) {
    const int k = i / NPOS, pos = i % NPOS;
    const int64_t ce = ce0 + k;
    T val = T(0);
    if (ce < cd.ne) {
      const int cx = (int)(ce % cd.ex);
      const int64_t t = ce / cd.ex;
      const int cy = (int)(t % cd.ey), cz = (int)(t / cd.ey);
      const int fx = cx * FCT + pos % FCT, fy = cy * FCT + pos / FCT % FCT, fz = cz * FCT + pos / (FCT * FCT);
      if (fx < fd.ex && fy < fd.ey && fz < fd.ez) {
        const int64_t fe = fx + (int64_t)fd.ex * (fy + (int64_t)fd.ey * fz);
        bool fixed = false;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const int64_t vv = (fx + (a & 1)) + (int64_t)fd.vx * ((fy + ((a >> 1) & 1)) + (int64_t)fd.vy * (fz + (a >> 2)));
          const uint8_t m = vmask[vv];
          fixed |= (m & 7) != 7;
        }
        val = fixed ? T(0) : T(rhop[fe]);
      }
    }
    rp[k][pos] = val;
  }
  __syncthreads();
  const int ent = threadIdx.x;
  if (ent >= 300) return;
  // upper-triangle index -> (i, j), i <= j
  int i = 0, rem = ent;
  while (rem >= 24 - i) { rem -= 24 - i; ++i; }
  const int j = i + rem;
  T acc[GAL_CE];
#pragma unroll
  for (int k = 0; k < GAL_CE; ++k) acc[k] = T(0);
  for (int pos = 0; pos < NPOS; ++pos) {
    const T tv = Ttab[pos * 576 + i * 24 + j];
#pragma unroll
    for (int k = 0; k < GAL_CE; ++k) acc[k] += rp[k][pos] * tv;
  }
#pragma unroll
  for (int k = 0; k < GAL_CE; ++k) {
    const int64_t ce = ce0 + k;
    if (ce >= cd.ne) break;
    kel[ce * 576 + i * 24 + j] = acc[k];
    kel[ce * 576 + j * 24 + i] = acc[k];
  }
}

// Fixed-DOF fine elements: K_E += Q^T Ktilde_e Q, one CTA per coarse element,
// one thread per entry; fine elements are visited in a fixed order.
template <typename T, int FCT>
__global__ void __launch_bounds__(576) k_galerkin_fixed(LevelDims fd, LevelDims cd,
                                                        const double* __restrict__ rhop,
                                                        const uint8_t* __restrict__ eactive,
                                                        const uint8_t* __restrict__ vmask,
                                                        const double* __restrict__ Ke,
                                                        const int* __restrict__ list,
                                                        T* __restrict__ kel) {
  // products in the operator's precision: FP32 for the FP32 preconditioner's
  // operators (the FP64 form is bound by GB300's FP64 pipe), FP64 for FP64
  constexpr int NP = FCT * FCT * FCT;  // fine elements in the coarse element
  __shared__ T sK[576];
  __shared__ T sQ[8][8];
  __shared__ uint8_t sfree[NP][24];
  __shared__ uint8_t sflag[NP];
  const int64_t ce = list[blockIdx.x];
  const int cx = (int)(ce % cd.ex);
  const int64_t t = ce / cd.ex;
  const int cy = (int)(t % cd.ey), cz = (int)(t / cd.ey);
  const int ent = threadIdx.x;
  const int R = ent / 24, S = ent % 24;
  const int A = R / 3, i = R % 3, B = S / 3, j = S % 3;
  // free-DOF pattern of every fine element at once (one thread each); the
  // fine elements with all 24 DOFs free are left to the GEMM pass
  if (ent < NP) {
    const int px = ent % FCT, py = ent / FCT % FCT, pz = ent / (FCT * FCT);
    const int fx = cx * FCT + px, fy = cy * FCT + py, fz = cz * FCT + pz;
    int flag = 0;
    if (fx < fd.ex && fy < fd.ey && fz < fd.ez && eactive[fx + (int64_t)fd.ex * (fy + (int64_t)fd.ey * fz)]) {
      for (int a = 0; a < 8; ++a) {
        const int64_t vv = (fx + (a & 1)) + (int64_t)fd.vx * ((fy + ((a >> 1) & 1)) + (int64_t)fd.vy * (fz + (a >> 2)));
        const uint8_t m = vmask[vv];
        for (int c = 0; c < 3; ++c) sfree[ent][3 * a + c] = (m >> c) & 1;
        if ((m & 7) != 7) flag = 1;
      }
    }
    sflag[ent] = (uint8_t)flag;
  }
  __syncthreads();
  T acc = T(0);
  for (int pos = 0; pos < NP; ++pos) {
    if (!sflag[pos]) continue;  // the same for the whole CTA
    const int px = pos % FCT, py = pos / FCT % FCT, pz = pos / (FCT * FCT);
    const int fx = cx * FCT + px, fy = cy * FCT + py, fz = cz * FCT + pz;
    const double pe = rhop[fx + (int64_t)fd.ex * (fy + (int64_t)fd.ey * fz)];
    {
      const int r = ent / 24, s2 = ent % 24;
      double k = pe * Ke[ent];
      if (!sfree[pos][r] || !sfree[pos][s2]) k = (r == s2) ? 1e6 : 0.0;
      sK[ent] = T(k);
    }
    if (ent < 64) {
      const int a = ent / 8, C = ent % 8;
      const int q[3] = {px + (a & 1), py + ((a >> 1) & 1), pz + (a >> 2)};
      const int cc[3] = {C & 1, (C >> 1) & 1, C >> 2};
      double w = 1.0;
      for (int k = 0; k < 3; ++k) w *= cc[k] ? (double)q[k] / FCT : (double)(FCT - q[k]) / FCT;
      sQ[a][C] = T(w);
    }
    __syncthreads();
    T s = T(0);
    for (int a = 0; a < 8; ++a) {
      const T qa = sQ[a][A];
      if (qa == T(0)) continue;
      T inner = T(0);
      for (int b = 0; b < 8; ++b) inner += sK[(3 * a + i) * 24 + 3 * b + j] * sQ[b][B];
      s += qa * inner;
    }
    acc += s;
    __syncthreads();  // sK and sQ are rewritten for the next fine element
  }
  if (acc != T(0)) kel[ce * 576 + ent] += acc;
}

// Dyadic Galerkin: K_E = sum_children Q_c^T K_child Q_c (grid/Grid.cu:839-896 in
// element form).  One CTA per coarse element, two-stage product per child.
template <typename T>
__global__ void __launch_bounds__(576) k_galerkin_dyadic(LevelDims fd, LevelDims cd,
                                                         const uint8_t* __restrict__ eactive_f,
                                                         const T* __restrict__ kel_f,
                                                         T* __restrict__ kel_c) {
  __shared__ T sK[576];
  __shared__ T sT[576];
  __shared__ T sQ[8][8];
  const int64_t ce = blockIdx.x;
  const int cx = (int)(ce % cd.ex);
  const int64_t t = ce / cd.ex;
  const int cy = (int)(t % cd.ey), cz = (int)(t / cd.ey);
  const int ent = threadIdx.x;
  const int R = ent / 24, S = ent % 24;
  T acc = T(0);
  for (int c = 0; c < 8; ++c) {
    const int ox = c & 1, oy = (c >> 1) & 1, oz = c >> 2;
    const int fx = 2 * cx + ox, fy = 2 * cy + oy, fz = 2 * cz + oz;
    const bool on = fx < fd.ex && fy < fd.ey && fz < fd.ez &&
                    eactive_f[fx + (int64_t)fd.ex * (fy + (int64_t)fd.ey * fz)];
    if (!on) continue;  // uniform across the CTA
    const int64_t fe = fx + (int64_t)fd.ex * (fy + (int64_t)fd.ey * fz);
    __syncthreads();
    sK[ent] = kel_f[fe * 576 + ent];
    if (ent < 64) {
      const int a = ent / 8, C = ent % 8;
      const int q[3] = {ox + (a & 1), oy + ((a >> 1) & 1), oz + (a >> 2)};
      const int cc[3] = {C & 1, (C >> 1) & 1, C >> 2};
      T w = T(1);
      for (int k = 0; k < 3; ++k) w *= cc[k] ? T(q[k]) / T(2) : T(2 - q[k]) / T(2);
      sQ[a][C] = w;
    }
    __syncthreads();
    {  // stage 1: sT[r][3C+jj] = sum_b K[r][3b+jj] Q[b][C]
      const int r = ent / 24, col = ent % 24, C = col / 3, jj = col % 3;
      T s = T(0);
#pragma unroll
      for (int b = 0; b < 8; ++b) s += sK[r * 24 + 3 * b + jj] * sQ[b][C];
      sT[ent] = s;
    }
    __syncthreads();
    {  // stage 2: acc[(A,i),S] += sum_a Q[a][A] T[3a+i][S]
      const int A = R / 3, i = R % 3;
      T s = T(0);
#pragma unroll
      for (int a = 0; a < 8; ++a) s += sQ[a][A] * sT[(3 * a + i) * 24 + S];
      acc += s;
    }
  }
  kel_c[ce * 576 + ent] = acc;
}

// Stencil assembly from element matrices: thread per (neighbour d, vertex v),
// consecutive threads along what the layout stores together; FP64 by vertex, a warp
// one neighbour of 32 vertices: its blocks are sums of as many elements (1 to 8)
// in every lane, which counts for more there than whole lines (operator update
// at 192x96x96, FP64 2,310 -> 2,284 us, FP32 358 -> 429).  planes: also the [243][nv]
// form that callers read (FP64, null: none).
template <typename T>
__global__ void k_assemble_stencil(LevelDims d, const uint8_t* __restrict__ eactive,
                                   const uint8_t* __restrict__ vmask, const T* __restrict__ kel,
                                   T* __restrict__ st, StIdx si, T* __restrict__ planes) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int k;
  int64_t v;
  if (sizeof(T) == 4 && si.form == 2) {
    v = gid / 27;
    k = (int)(gid - 27 * v);
    if (v >= d.nv) return;
  } else if (si.form == 2) {
    const int64_t w = gid >> 5, g = w / 27;
    k = (int)(w - 27 * g);
    v = 32 * g + (gid & 31);
    if (v >= d.nv) return;
  } else {
    if (gid >= 27 * d.nv) return;
    k = (int)(gid / d.nv);
    v = gid % d.nv;
  }
  const int x = (int)(v % d.vx);
  const int64_t t = v / d.vx;
  const int y = (int)(t % d.vy), z = (int)(t / d.vy);
  const int dx = k % 3 - 1, dy = k / 3 % 3 - 1, dz = k / 9 - 1;
  T blk[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) blk[q] = T(0);
  // elements containing both v and v+(dx,dy,dz)
  for (int ez = z - 1; ez <= z; ++ez) {
    if (ez < 0 || ez >= d.ez) continue;
    const int az = z - ez, bz = az + dz;
    if (bz < 0 || bz > 1) continue;
    for (int ey = y - 1; ey <= y; ++ey) {
      if (ey < 0 || ey >= d.ey) continue;
      const int ay = y - ey, by = ay + dy;
      if (by < 0 || by > 1) continue;
      for (int ex = x - 1; ex <= x; ++ex) {
        if (ex < 0 || ex >= d.ex) continue;
        const int ax = x - ex, bx = ax + dx;
        if (bx < 0 || bx > 1) continue;
        const int64_t e = ex + (int64_t)d.ex * (ey + (int64_t)d.ey * ez);
        if (!eactive[e]) continue;
        const int a = ax + 2 * ay + 4 * az, b = bx + 2 * by + 4 * bz;
        const T* K = kel + e * 576;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) blk[3 * i + j] += K[(3 * a + i) * 24 + 3 * b + j];
      }
    }
  }
  if (k == 13 && !(vmask[v] & 8)) {
    blk[0] = T(1); blk[4] = T(1); blk[8] = T(1);
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    st[si.base(v) + k * si.ks() + q * si.es()] = blk[q];
    if (planes) planes[(int64_t)(k * 9 + q) * d.nv + v] = blk[q];
  }
}

__global__ void k_stencil_planes(int64_t nv, const double* __restrict__ st, StIdx si, double* __restrict__ planes) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= 243 * nv) return;
  const int64_t q = gid / nv, v = gid - q * nv;
  planes[gid] = st[si.base(v) + q / 9 * si.ks() + q % 9 * si.es()];
}

template <typename T>
__global__ void k_dense_from_stencil(LevelDims d, const T* __restrict__ st, StIdx si, double* __restrict__ A) {
  const int64_t n = 3 * d.nv;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= 243 * d.nv) return;
  const int64_t v = gid / 243;
  const int q = (int)(gid - v * 243), e = q / 27, k = q - 27 * e, i = e / 3, j = e - 3 * i;
  const int x = (int)(v % d.vx);
  const int64_t t = v / d.vx;
  const int y = (int)(t % d.vy), z = (int)(t / d.vy);
  const int nx = x + k % 3 - 1, ny = y + k / 3 % 3 - 1, nz = z + k / 9 - 1;
  if (nx < 0 || ny < 0 || nz < 0 || nx >= d.vx || ny >= d.vy || nz >= d.vz) return;
  const int64_t nb = nx + (int64_t)d.vx * (ny + (int64_t)d.vy * nz);
  A[(3 * v + i) * n + 3 * nb + j] = (double)st[si.base(v) + k * si.ks() + e * si.es()];
}

__global__ void k_symmetrize(int n, double* A) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)n * n) return;
  const int i = (int)(gid / n), j = (int)(gid % n);
  if (j >= i) return;
  const double s = 0.5 * (A[(int64_t)i * n + j] + A[(int64_t)j * n + i]);
  A[(int64_t)i * n + j] = s;
  A[(int64_t)j * n + i] = s;
}

// Blocked Gauss-Jordan inversion (in place, SPD matrix), for matrices too large
// for k_gj_sweep.  A pivot below 1e-10 of the largest diagonal entry belongs to
// a null direction (a floating part of the domain): its row and column are
// dropped, which gives the inverse of the remaining DOFs, as the reference's
// pseudo-inverse does for its coarsest system (grid/Grid.cpp:3657, 4072).
// status[0] counts dropped pivots; a clearly negative pivot sets status[1] = k+1
// and every block stops at the same step.  For each panel K of GJB pivots: one CTA inverts the
// diagonal block D = A[K,K] pivot by pivot in shared memory (dropping pivots
// <= tol); all CTAs form the row panel P = D^-1 A[K,:] and copy the column panel
// C = A[:,K]; then every element gets its rank-GJB update
//   A[i,c] = D^-1 | P | -C D^-1 | A[i,c] - C[i,:] P[:,c]
// for (i in K, c in K) | (i in K) | (c in K) | otherwise.  Three grid barriers
// per panel instead of two per pivot.
constexpr int GJB = 32;

//
// DFC: the rank-GJB updates of phase C (n^3 of the n^3 + O(n^2 GJB) work) run
// in double-float arithmetic on the FP32 pipe (58x the FP64 rate on GB300),
// with the panels split into (hi, lo) floats once per panel; the panel
// factorisation stays FP64, where its serial latency matters more than its
// rate.  Used when the coarsest matrix comes from FP32 stencils.  (Measured
// at n = 1617, 304 CTAs: splitting the panels as each tile is staged kept the
// FP64 pipe 55% busy with conversions, 6.6 ms against 5.2 ms; also holding the
// matrix split in place for the whole inversion took the FP64 pipe to 18% but
// ran 5.4 ms, and the update on packed two-lane FP32 instructions cut the
// instructions by a quarter but ran 5.6 ms: the panel barriers and the serial
// panel work then set the pace.)
// (No __restrict__ on what the CTAs hand each other between grid barriers: it
// lets the compiler keep a value across a barrier.)
template <bool DFC>
__global__ void __launch_bounds__(256) k_gj_blocked(int n, double* A, double* work, int* status) {
  cg::grid_group grid = cg::this_grid();
  __shared__ double sd[GJB][GJB + 1];
  __shared__ df scd[DFC ? GJB : 1][GJB + 1];
  __shared__ df spd[DFC ? GJB : 1][GJB + 1];
  __shared__ double sc[GJB][GJB + 1];
  __shared__ double sp[GJB][GJB + 1];
  double* P = work + GJB * GJB;      // [GJB][n]
  double* Cp = P + (int64_t)GJB * n; // [n][GJB]
  df* Pdf = reinterpret_cast<df*>(Cp + (int64_t)GJB * n);  // P split, [GJB][n]
  df* Cdf = Pdf + (int64_t)GJB * n;                          // Cp split, [n][GJB]
  const int tid = threadIdx.x;
  double dmax = 0.0;
  for (int k = 0; k < n; ++k) dmax = fmax(dmax, fabs(A[(int64_t)k * n + k]));
  const double tol = 1e-10 * dmax;
  const int nblk_tiles = (n + GJB - 1) / GJB;
  // ---- A: CTA 0 inverts a diagonal block D = A[K,K] (K = [k0, k0 + GJB)) in
  // FP64 and publishes it through the work array.  The block of panel k + 1
  // is inverted during panel k's update (look-ahead): CTA 0 updates that one
  // tile first and inverts it while the other CTAs update the rest.
  // (Measured alternatives on GB300 at n = 675: every CTA inverting its own
  // copy saves a grid barrier but ran at 2.4 ms in FP64, every SM's narrow
  // FP64 pipe then carrying the panel work, and at 2.6 ms in double-float,
  // whose pivot steps lengthen the serial chain; inverting between the update
  // phases, with its own grid barrier, ran at 1.9 ms; this form at 1.56 ms.)
  auto panel_invert = [&](int k0) {
    const int kb = min(GJB, n - k0);
    for (int e = tid; e < GJB * GJB; e += blockDim.x) {
      const int r = e / GJB, c = e % GJB;
      sd[r][c] = (r < kb && c < kb) ? A[(int64_t)(k0 + r) * n + k0 + c] : 0.0;
    }
    __syncthreads();
    for (int j = 0; j < kb; ++j) {
      const double p = sd[j][j];
      if (p < -tol) {
        if (tid == 0) status[1] = k0 + j + 1;
        break;
      }
      __syncthreads();
      if (p <= tol) {  // drop DOF k0 + j
        for (int e = tid; e < 2 * GJB; e += blockDim.x) {
          if (e < GJB) sd[j][e] = 0.0;
          else sd[e - GJB][j] = 0.0;
        }
        if (tid == 0) status[0] += 1;
        __syncthreads();
        continue;
      }
      // 1/p: FP32 estimate refined by two Newton steps r <- r + r (1 - p r)
      double rp = (double)__frcp_rn((float)p);
      rp = fma(rp, fma(-p, rp, 1.0), rp);
      rp = fma(rp, fma(-p, rp, 1.0), rp);
      for (int e = tid; e < GJB * GJB; e += blockDim.x) {
        const int r = e / GJB, c = e % GJB;
        if (r < kb && c < kb && r != j && c != j) sd[r][c] -= sd[r][j] * sd[j][c] * rp;
      }
      __syncthreads();
      for (int e = tid; e < 2 * kb; e += blockDim.x) {
        if (e < kb) { if (e != j) sd[j][e] *= rp; else sd[j][j] = rp; }
        else { const int r = e - kb; if (r != j) sd[r][j] *= -rp; }
      }
      __syncthreads();
    }
    __syncthreads();
    for (int e = tid; e < GJB * GJB; e += blockDim.x) work[e] = sd[e / GJB][e % GJB];
  };
  if (blockIdx.x == 0) panel_invert(0);
  grid.sync();
  for (int k0 = 0; k0 < n; k0 += GJB) {
    const int kb = min(GJB, n - k0);
    // indefinite pivot: every thread of every CTA has to see it, or the others
    // wait for this one at the next barrier
    if (*(volatile int*)(status + 1)) return;
    for (int e = tid; e < GJB * GJB; e += blockDim.x) sd[e / GJB][e % GJB] = work[e];
    __syncthreads();
    // ---- B: row panel P = D^-1 A[K,:] (columns outside K) and column panel C = A[:,K]
    const int64_t gt = (int64_t)blockIdx.x * blockDim.x + tid, gs = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = gt; e < (int64_t)kb * n; e += gs) {
      const int r = (int)(e / n), c = (int)(e % n);
      double v = 0.0;
      if (c < k0 || c >= k0 + kb) {
#pragma unroll 8
        for (int m = 0; m < kb; ++m) v += sd[r][m] * A[(int64_t)(k0 + m) * n + c];
      }
      P[(int64_t)r * n + c] = v;
      if constexpr (DFC) Pdf[(int64_t)r * n + c] = df_from(v);
    }
    for (int64_t e = gt; e < (int64_t)n * kb; e += gs) {
      const int i = (int)(e / kb), m = (int)(e % kb);
      const double v = (i < k0 || i >= k0 + kb) ? A[(int64_t)i * n + k0 + m] : 0.0;
      Cp[(int64_t)i * GJB + m] = v;
      if constexpr (DFC) Cdf[(int64_t)i * GJB + m] = df_from(v);
    }
    grid.sync();
    // ---- C: rank-kb update, GJB x GJB tiles of A.  With a next panel, CTA 0
    // takes only its diagonal tile and then inverts it; the others share the
    // rest.
    const int k1 = k0 + GJB, tn = k1 < n ? (k1 / GJB) * (nblk_tiles + 1) : -1;
    const bool ahead = tn >= 0 && gridDim.x > 1;
    const int t_first = ahead ? (blockIdx.x == 0 ? tn : (int)blockIdx.x - 1) : (int)blockIdx.x;
    const int t_step = ahead ? (blockIdx.x == 0 ? nblk_tiles * nblk_tiles : (int)gridDim.x - 1) : (int)gridDim.x;
    for (int t0 = t_first; t0 < nblk_tiles * nblk_tiles; t0 += t_step) {
      // the CTAs other than 0 skip the diagonal tile of the next panel
      const int t = (ahead && blockIdx.x != 0 && t0 >= tn) ? t0 + 1 : t0;
      if (t >= nblk_tiles * nblk_tiles) break;
      const int ti = (t / nblk_tiles) * GJB, tc = (t % nblk_tiles) * GJB;
      // a tile outside the panel's rows and columns: every element gets the update
      const bool band = (ti < k0 + kb && ti + GJB > k0) || (tc < k0 + kb && tc + GJB > k0);
      __syncthreads();
      for (int e = tid; e < GJB * GJB; e += blockDim.x) {
        const int r = e / GJB, c = e % GJB;
        const bool inc = ti + r < n && c < kb, inp = r < kb && tc + c < n;
        if (!DFC || band) {
          sc[r][c] = inc ? Cp[(int64_t)(ti + r) * GJB + c] : 0.0;
          sp[r][c] = inp ? P[(int64_t)r * n + tc + c] : 0.0;
        }
        if constexpr (DFC) {
          scd[r][c] = inc ? Cdf[(int64_t)(ti + r) * GJB + c] : df(0.f, 0.f);
          spd[r][c] = inp ? Pdf[(int64_t)r * n + tc + c] : df(0.f, 0.f);
        }
      }
      __syncthreads();
      if (!band && blockDim.x == 8 * GJB) {
        // four rows of one column per thread: four independent chains share
        // each panel value (per element the operations and order of the loop
        // below)
        const int c = tid % GJB, r0 = tid / GJB, col = tc + c;
        double* a[4];
        bool in[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = ti + r0 + 8 * q;
          in[q] = i < n && col < n;
          a[q] = A + (int64_t)(in[q] ? i : 0) * n + (in[q] ? col : 0);
        }
        if constexpr (DFC) {
          df v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) v[q] = df_from(in[q] ? *a[q] : 0.0);
#pragma unroll 4
          for (int m = 0; m < kb; ++m) {
            const df pm = spd[m][c];
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = v[q] - scd[r0 + 8 * q][m] * pm;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (in[q]) *a[q] = df_to(v[q]);
        } else {
          double v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) v[q] = in[q] ? *a[q] : 0.0;
#pragma unroll 4
          for (int m = 0; m < kb; ++m) {
            const double pm = sp[m][c];
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] -= sc[r0 + 8 * q][m] * pm;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (in[q]) *a[q] = v[q];
        }
        continue;
      }
      for (int e = tid; e < GJB * GJB; e += blockDim.x) {
        const int r = e / GJB, c = e % GJB;
        const int i = ti + r, col = tc + c;
        if (i >= n || col >= n) continue;
        const bool iK = i >= k0 && i < k0 + kb, cK = col >= k0 && col < k0 + kb;
        double& a = A[(int64_t)i * n + col];
        if (iK && cK) {
          a = sd[i - k0][col - k0];
        } else if (iK) {
          a = sp[i - k0][c];
        } else if (cK) {
          double v = 0.0;
          for (int m = 0; m < kb; ++m) v += sc[r][m] * sd[m][col - k0];
          a = -v;
        } else if constexpr (DFC) {
          df v = df_from(a);
          for (int m = 0; m < kb; ++m) v = v - scd[r][m] * spd[m][c];
          a = df_to(v);
        } else {
          double v = a;
          for (int m = 0; m < kb; ++m) v -= sc[r][m] * sp[m][c];
          a = v;
        }
      }
    }
    if (k1 < n && blockIdx.x == 0) {
      __syncthreads();  // the tile's updates are visible to the whole CTA
      panel_invert(k1);
    }
    grid.sync();
  }
}

// ---------------------------------------------------------------------------
// Inversion of the coarsest matrix by symmetric sweeps, the lower triangle held
// on chip.  Sweeping a panel K of 32 pivots maps a symmetric A to
//   A_KK <- -A_KK^-1,  A_iK <- W_i = A_iK A_KK^-1,  A_ij <- A_ij - W_i A_Kj,
// which is symmetric again, and sweeping every panel leaves -A^-1, so only the
// 32 x 32 tiles (i, j), i >= j, are kept: half the rank-32 updates of
// Gauss-Jordan on the full matrix.  Each CTA owns consecutive tiles of that
// triangle in shared memory for the whole inversion (n = 1617: nine tiles a
// SM, n = 675: two), so a panel moves only the panel itself through L2:
//   B: W_j = C_j D^-1, the panel's rows dealt evenly over all CTAs, with
//      C_j = A_jK and D = A_KK published by the phase before;
//   C: every tile's update; the owners of the next panel's tiles publish them.
// CTA 0 owns no tile: during C it forms the next diagonal tile from the
// published parts and inverts it.  Two grid barriers a panel.
// Precision: tiles and updates are double-float, as the updates of
// k_gj_blocked<true> are (an FP64 tile between two of them holds no more).  The
// panel has FP64 accuracy, as there: the block's inverse X is formed in
// double-float, where its pivots' serial chain is short, and B corrects
// W0 = C_j X by the FP64 residual C_j - W0 D, which takes X's error squared; for
// j = K that refines the inverse itself.  Error of the inverse on matrices of
// designs, this / k_gj_blocked<true> / panels in double-float: n = 24 6.4e-16 /
// 8.8e-16 / 1.8e-14, 36 2.5e-14 / 2.3e-14 / 1.3e-13, 135 0.9e-13 / 3.3e-13 /
// 5.6e-13, 675 2.0e-13 / 6.7e-13 / 7.5e-13, 1617 2.9e-14 / 1.9e-13 / 1.9e-13
// (the updates' terms are summed apart from the element).
// Bounds: at n = 675 the chain of a panel (C for the diagonal tile 3 us, its
// inversion 7 us, B 5 us, barriers 2.5 us), at n = 1617 the updates (480 FP32
// instructions an element and panel) and B's FP64 products (2.7 us of 4 us a
// panel).  Inversion alone, this / k_gj_blocked<true> / panels in double-float:
// n = 135 0.13 / 0.30 / 0.10 ms, 336 0.24 / 0.67 / 0.19, 675 0.45 / 1.51 / 0.37,
// 1617 1.90 / 5.23 / 1.66, 2520 6.1 / 17.2 / 5.3.  (The block's pivots in FP64
// too: 0.67 ms at n = 675.)
// The pivot-drop rule and status are k_gj_blocked's.
// ---------------------------------------------------------------------------
constexpr int GJT = GJB * GJB;         // elements of a tile
constexpr int GJP = GJB + 1;           // pitch of a tile row in shared memory
constexpr int GJ_TILE = GJB * GJP;     // shared elements of an owned tile
constexpr int GJ_THREADS = 512;
constexpr int SB = 4;                  // pivots a step of the diagonal block's inversion
constexpr int GJ_SWEEP_SMEM = 212 * 1024;  // dynamic shared memory a CTA may take (227 KB less the static arrays)

__device__ __forceinline__ df df_ldcg(const df* p) {
  const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
  return df(v.x, v.y);
}
__device__ __forceinline__ df df_shfl(df v, int l) {
  return df(__shfl_sync(0xffffffffu, v.hi, l), __shfl_sync(0xffffffffu, v.lo, l));
}
__device__ __forceinline__ df df_neg(df v) { return df(-v.hi, -v.lo); }
// acc - a b: TwoProd, TwoSum and one renormalisation
__device__ __forceinline__ df df_nfma(df acc, df a, df b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  const float t = __fsub_rn(acc.hi, p), z = __fsub_rn(t, acc.hi);
  const float r = __fsub_rn(__fsub_rn(acc.hi, __fsub_rn(t, z)), __fadd_rn(p, z));
  return df_fast2sum(t, __fadd_rn(r, __fsub_rn(acc.lo, e)));
}
// 1/p: FP32 estimate, one Newton step with its second-order term
__device__ __forceinline__ df df_rcp(df p) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(p.hi));
  const float e = __fmaf_rn(-p.lo, r, __fmaf_rn(-p.hi, r, 1.f));
  return df_fast2sum(r, __fmul_rn(r, __fmaf_rn(e, e, e)));
}

// Inverts the kb x kb symmetric block T (pitch GJP, lower triangle; rows and
// columns from kb on are zero) and writes the full inverse to out[GJT] and the
// block itself in FP64 to d64[GJT].  Called by all threads of a CTA.  k0: index
// of the first pivot (status).
// Four pivots at a time: warp 0 sweeps them on their own four columns, held in
// registers (lane r: row r), so a pivot costs shuffles and arithmetic but no
// barrier, and the other elements then get their rank-4 update from all warps.
// (One barrier a pivot took twice as long.)
__device__ __forceinline__ void sweep_block(const df* T, df (*sd)[GJP], df (*sv)[SB][GJB], int kb, int k0, df tol,
                                            int* status, df* out, double* d64) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const df zero(0.f, 0.f);
  for (int e = tid; e < GJT; e += GJ_THREADS) sd[e / GJB][e % GJB] = T[(e / GJB) * GJP + e % GJB];
  // this thread's element of the lower triangle with the four panel rows taken
  // out: rows r and 27 - r of that 28-row triangle together hold 29
  constexpr int R = GJB - SB;
  static_assert((R / 2) * (R + 1) <= GJ_THREADS, "one element a thread");
  const int pr = tid / (R + 1), pk = tid - pr * (R + 1);
  const bool mine = tid < (R / 2) * (R + 1);
  const int r28 = pk <= pr ? pr : R - 1 - pr, c28 = pk <= pr ? pk : pk - pr - 1;
  for (int j = 0; j < kb; j += SB) {
    __syncthreads();
    if (warp == 0) {
      df v[SB];
#pragma unroll
      for (int q = 0; q < SB; ++q) v[q] = lane >= j + q ? sd[lane][j + q] : sd[j + q][lane];
#pragma unroll
      for (int q = 0; q < SB; ++q) {
        if (j + q >= kb) {
          sv[0][q][lane] = sv[1][q][lane] = zero;
          continue;
        }
        const df p = df_shfl(v[q], j + q);
        const bool drop = p.hi < tol.hi || (p.hi == tol.hi && p.lo <= tol.lo);
        df rp = df_rcp(p);
        if (drop) rp = zero;
        const df w = drop ? zero : v[q] * rp;
        const df m = lane == j + q ? df_neg(rp) : w;  // the swept column; the pivot row gets 0 - (-rp) a
        sv[0][q][lane] = v[q];
        sv[1][q][lane] = m;
#pragma unroll
        for (int i = 0; i < SB; ++i) {
          if (i == q) continue;
          const df s = df_shfl(v[q], j + i);
          v[i] = df_nfma(lane == j + q ? zero : v[i], m, s);
        }
        v[q] = m;
        if (drop && lane == 0) {
          if (p.hi < -tol.hi || (p.hi == -tol.hi && p.lo < -tol.lo)) status[1] = k0 + j + q + 1;
          else status[0] += 1;
        }
      }
#pragma unroll
      for (int q = 0; q < SB; ++q)
        if (lane >= j + q) sd[lane][j + q] = v[q];
        else if (lane < j) sd[j + q][lane] = v[q];
    } else if (j == 0) {  // (the warps that wait for the first pivots)
      for (int e = tid - 32; e < GJT; e += GJ_THREADS - 32) {
        const int r = e / GJB, c = e % GJB;
        d64[e] = df_to(r >= c ? T[r * GJP + c] : T[c * GJP + r]);
      }
    }
    __syncthreads();
    if (mine) {
      const int r = r28 < j ? r28 : r28 + SB, c = c28 < j ? c28 : c28 + SB;
      df x = sd[r][c];
#pragma unroll
      for (int q = 0; q < SB; ++q) x = df_nfma(x, sv[1][q][r], sv[0][q][c]);
      sd[r][c] = x;
    }
  }
  __syncthreads();
  for (int e = tid; e < GJT; e += GJ_THREADS) {
    const int r = e / GJB, c = e % GJB;
    out[e] = df_neg(r >= c ? sd[r][c] : sd[c][r]);
  }
}

__global__ void __launch_bounds__(GJ_THREADS, 1) k_gj_sweep(int n, double* A, float* A32, double* work, int* status) {
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) unsigned char gj_smem[];
  df* sW = reinterpret_cast<df*>(gj_smem);  // [2][GJT] staged W_i, [r][m]
  df* sC = sW + 2 * GJT;                   // [2][GJT] staged C_j transposed, [m][c]
  df* sT = sC + 2 * GJT;                   // owned tiles [r][c], pitch GJP
  __shared__ df sd[GJB][GJP];
  __shared__ df sv[2][SB][GJB];
  __shared__ double smax[GJ_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = (n + GJB - 1) / GJB;
  // published panels: C_j transposed ([2][nt][m][r]), W_j ([nt][r][m], the
  // block's inverse for j = K), the block before its refinement, the block itself
  // in FP64, the last block's inverse in FP64, and the next but one diagonal
  // tile ([2])
  df* Cg = reinterpret_cast<df*>(work);
  df* Wg = Cg + (int64_t)2 * nt * GJT;
  df* Xg = Wg + (int64_t)nt * GJT;
  double* D64 = reinterpret_cast<double*>(Xg + GJT);
  double* X64 = D64 + GJT;
  df* Qg = reinterpret_cast<df*>(X64 + GJT);
  double dmax = 0.0;
  for (int k = tid; k < n; k += GJ_THREADS) dmax = fmax(dmax, fabs(A[(int64_t)k * n + k]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
  if (lane == 0) smax[warp] = dmax;
  __syncthreads();
  for (int k = 0; k < GJ_THREADS / 32; ++k) dmax = fmax(dmax, smax[k]);
  const df tol = df_from(1e-10 * dmax);
  // tiles t0 .. t1 of the triangle in row order; CTA 0 has none unless alone
  const int nb = (int)gridDim.x, own = nb > 1 ? nb - 1 : 1, me = nb > 1 ? (int)blockIdx.x - 1 : 0;
  const int64_t ntri = (int64_t)nt * (nt + 1) / 2;
  const int t0 = me < 0 ? 0 : (int)(ntri * me / own), t1 = me < 0 ? 0 : (int)(ntri * (me + 1) / own);
  int i0 = (int)((sqrtf(8.f * (float)t0 + 1.f) - 1.f) * 0.5f);
  while ((i0 + 1) * (i0 + 2) / 2 <= t0) ++i0;
  while (i0 * (i0 + 1) / 2 > t0) --i0;
  const int j0 = t0 - i0 * (i0 + 1) / 2;
  // publishes tile (i, j) where panel q or the diagonal after it needs it
  auto publish = [&](const df* T, int i, int j, int q) {
    if (q < nt && (i == q) != (j == q)) {  // C_m transposed, m the other index
      df* dst = Cg + ((int64_t)(q & 1) * nt + (i == q ? j : i)) * GJT;
      for (int e = tid; e < GJT; e += GJ_THREADS) {
        const int m = e / GJB, r = e % GJB;
        dst[e] = T[i == q ? m * GJP + r : r * GJP + m];
      }
    }
    if (i == j && i == q + 1)
      for (int e = tid; e < GJT; e += GJ_THREADS) Qg[(i & 1) * GJT + e] = T[(e / GJB) * GJP + e % GJB];
  };
  // the symmetric part of A, as k_symmetrize forms it
  auto entry = [&](int r, int c) { return r < n && c < n ? 0.5 * (A[(int64_t)r * n + c] + A[(int64_t)c * n + r]) : 0.0; };
  {
    int i = i0, j = j0;
    for (int t = t0; t < t1; ++t) {
      df* T = sT + (int64_t)(t - t0) * GJ_TILE;
      for (int e = tid; e < GJT; e += GJ_THREADS)
        T[(e / GJB) * GJP + e % GJB] = df_from(entry(i * GJB + e / GJB, j * GJB + e % GJB));
      __syncthreads();
      publish(T, i, j, 0);
      if (++j > i) { ++i; j = 0; }
    }
  }
  df* sQ = nb > 1 ? sT : sC;  // CTA 0's diagonal tile (it owns none, or the panels have not begun)
  if (blockIdx.x == 0) {
    for (int e = tid; e < GJT; e += GJ_THREADS) sQ[(e / GJB) * GJP + e % GJB] = df_from(entry(e / GJB, e % GJB));
    __syncthreads();
    sweep_block(sQ, sd, sv, min(GJB, n), 0, tol, status, Xg, D64);
  }
  grid.sync();
  for (int k = 0; k < nt; ++k) {
    if (__ldcg(status + 1)) return;  // indefinite pivot: every CTA sees it after the barrier
    const df* Ck = Cg + (int64_t)(k & 1) * nt * GJT;
    // ---- B: W_j = C_j D^-1, the panel's rows dealt evenly over the CTAs, a warp
    // a row (lane m holds C_j(r, m), then W_j(r, m)): W0 = C_j X with the block's
    // inverse X as it came, the residual C_j - W0 D in FP64, W = W0 + residual X.
    // For j = K, C is the identity and W the inverse itself.
    const int rows = nt * GJB, per = (rows + nb - 1) / nb, r0 = (int)blockIdx.x * per, r1 = min(rows, r0 + per);
    if (r0 < r1) {
      df* X = sW;
      double* D = reinterpret_cast<double*>(sW + GJT);
      auto load_c = [&](int g) {
        return g / GJB == k ? df(lane == g % GJB ? 1 : 0) : df_ldcg(Ck + (int64_t)(g / GJB) * GJT + lane * GJB + g % GJB);
      };
      df cn = r0 + warp < r1 ? load_c(r0 + warp) : df(0);  // in flight with the block
#pragma unroll
      for (int q = 0; q < GJT / GJ_THREADS; ++q) {
        X[tid + q * GJ_THREADS] = df_ldcg(Xg + tid + q * GJ_THREADS);
        D[tid + q * GJ_THREADS] = __ldcg(D64 + tid + q * GJ_THREADS);
      }
      __syncthreads();
      for (int g = r0 + warp; g < r1; g += GJ_THREADS / 32) {
        const int j = g / GJB, r = g % GJB;
        const df c = cn;
        if (g + GJ_THREADS / 32 < r1) cn = load_c(g + GJ_THREADS / 32);
        df a[4] = {df(0), df(0), df(0), df(0)};  // four chains of each sum
#pragma unroll 2
        for (int m = 0; m < GJB; m += 4)
#pragma unroll
          for (int i = 0; i < 4; ++i) a[i] = df_nfma(a[i], df_shfl(c, m + i), X[(m + i) * GJB + lane]);
        const double w = -df_to((a[0] + a[1]) + (a[2] + a[3]));
        double e[4] = {df_to(c), 0.0, 0.0, 0.0};
#pragma unroll 2
        for (int m = 0; m < GJB; m += 4)
#pragma unroll
          for (int i = 0; i < 4; ++i) e[i] = fma(-__shfl_sync(0xffffffffu, w, m + i), D[(m + i) * GJB + lane], e[i]);
        const float res = (float)((e[0] + e[1]) + (e[2] + e[3]));
        float p = 0.f, q = 0.f;
#pragma unroll 4
        for (int m = 0; m < GJB; m += 2) {
          p = fmaf(__shfl_sync(0xffffffffu, res, m), X[m * GJB + lane].hi, p);
          q = fmaf(__shfl_sync(0xffffffffu, res, m + 1), X[(m + 1) * GJB + lane].hi, q);
        }
        const double v = w + (double)(p + q);
        Wg[(int64_t)j * GJT + r * GJB + lane] = df_from(v);
        if (k + 1 == nt && j == k) X64[r * GJB + lane] = v;
      }
    }
    grid.sync();
    // ---- C: the tiles' updates; CTA 0 inverts the next diagonal block
    const int k1 = k + 1;
    auto stage = [&](int buf, int i, int j) {
      const char* w = reinterpret_cast<const char*>(Wg + (int64_t)i * GJT);
      const char* c = reinterpret_cast<const char*>(Ck + (int64_t)j * GJT);
      const unsigned dw = (unsigned)__cvta_generic_to_shared(sW + buf * GJT), dc = (unsigned)__cvta_generic_to_shared(sC + buf * GJT);
      static_assert(GJT * 8 == GJ_THREADS * 16, "one 16-byte copy a thread and operand");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dw + tid * 16), "l"(w + tid * 16));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dc + tid * 16), "l"(c + tid * 16));
    };
    // T -= W C^T for the staged pair; two rows of one column a thread
    auto update = [&](df* T, int buf) {
      const df* W = sW + buf * GJT + warp * GJB;
      const df* C = sC + buf * GJT + lane;
      df* t = T + warp * GJP + lane;
      df v0(0), v1(0), w0(0), w1(0);  // even and odd m apart, and from the element: smaller sums, smaller error
#pragma unroll 4
      for (int m = 0; m < GJB; m += 2) {
        const df c = C[m * GJB], e = C[(m + 1) * GJB];
        v0 = df_nfma(v0, W[m], c);
        v1 = df_nfma(v1, W[16 * GJB + m], c);
        w0 = df_nfma(w0, W[m + 1], e);
        w1 = df_nfma(w1, W[16 * GJB + m + 1], e);
      }
      t[0] = t[0] + (v0 + w0);
      t[16 * GJP] = t[16 * GJP] + (v1 + w1);
    };
    if (blockIdx.x == 0 && k1 < nt) {
      stage(0, k1, k1);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      for (int e = tid; e < GJT; e += GJ_THREADS) sQ[(e / GJB) * GJP + e % GJB] = df_ldcg(Qg + (k1 & 1) * GJT + e);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
      update(sQ, 0);
      __syncthreads();
      sweep_block(sQ, sd, sv, min(GJB, n - k1 * GJB), k1 * GJB, tol, status, Xg, D64);
    }
    int i = i0, j = j0;
    if (t0 < t1 && i != k && j != k) stage(0, i, j);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int t = t0; t < t1; ++t) {
      const int buf = (t - t0) & 1, in = j + 1 > i ? i + 1 : i, jn = j + 1 > i ? 0 : j + 1;
      if (t + 1 < t1 && in != k && jn != k) stage(buf ^ 1, in, jn);
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;\n" ::: "memory");
      __syncthreads();
      df* T = sT + (int64_t)(t - t0) * GJ_TILE;
      if (i != k && j != k) {
        update(T, buf);
      } else if (i == j) {  // -D^-1
        for (int e = tid; e < GJT; e += GJ_THREADS)
          T[(e / GJB) * GJP + e % GJB] = df_neg(df_ldcg(Wg + (int64_t)k * GJT + e));
      } else {  // W_i, or W_j transposed
        const df* W = Wg + (int64_t)(j == k ? i : j) * GJT;
        for (int e = tid; e < GJT; e += GJ_THREADS) {
          const int a = e / GJB, b = e % GJB;
          T[j == k ? a * GJP + b : b * GJP + a] = df_ldcg(W + e);
        }
      }
      __syncthreads();
      publish(T, i, j, k1);
      i = in;
      j = jn;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    grid.sync();
  }
  // ---- A <- the inverse, both triangles, and its FP32 copy (the last block,
  // which no update followed, as it was formed in FP64)
  int i = i0, j = j0;
  for (int t = t0; t < t1; ++t) {
    const df* T = sT + (int64_t)(t - t0) * GJ_TILE;
    const bool lastb = i == nt - 1 && j == i;
    for (int e = tid; e < GJT; e += GJ_THREADS) {
      const int a = e / GJB, b = e % GJB;
      int r = i * GJB + a, c = j * GJB + b;
      if (r < n && c < n && (i != j || r >= c)) {
        const double v = lastb ? __ldcg(X64 + e) : -df_to(T[a * GJP + b]);
        A[(int64_t)r * n + c] = v;
        A32[(int64_t)r * n + c] = (float)v;
      }
      r = i * GJB + b;
      c = j * GJB + a;
      if (r < n && c < n && (i != j || r > c)) {
        const double v = lastb ? __ldcg(X64 + b * GJB + a) : -df_to(T[b * GJP + a]);
        A[(int64_t)c * n + r] = v;
        A32[(int64_t)c * n + r] = (float)v;
      }
    }
    if (++j > i) { ++i; j = 0; }
  }
}

__global__ void k_to_float(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

// u_soa = Ainv * f_soa over the dense DOF ordering 3v+c; one warp per row.
template <typename T>
__global__ void k_dense_gemv(int n, const T* __restrict__ Ainv, const T* __restrict__ f, T* __restrict__ u,
                             int64_t nv) {
  f += (int64_t)blockIdx.y * 3 * nv;  // right-hand side of the batch
  u += (int64_t)blockIdx.y * 3 * nv;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  T s = T(0);
  for (int j = lane; j < n; j += 32) s += Ainv[(int64_t)warp * n + j] * f[(j % 3) * nv + j / 3];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) u[(warp % 3) * nv + warp / 3] = s;
}

void launch_galerkin_first_impl(cudaStream_t s, const LevelDims& fd, const LevelDims& cd,
                                const double* rhop, const uint8_t* eactive_f, const uint8_t* vmask_f,
                                const double* Ttab64, const float* Ttab32, const double* Ke,
                                const int* fixed_list, int nfixed, double* kel, float* kel32) {
  const unsigned g = nblk(cd.ne, GAL_CE);
  const unsigned nf = (unsigned)nfixed;
  if (cd.factor == 4) {
    if (kel) {
      k_galerkin_gemm<double, 4><<<g, GAL_THREADS, 0, s>>>(fd, cd, rhop, vmask_f, Ttab64, kel);
      if (nf) k_galerkin_fixed<double, 4><<<nf, 576, 0, s>>>(fd, cd, rhop, eactive_f, vmask_f, Ke, fixed_list, kel);
    }
    if (kel32) {
      k_galerkin_gemm<float, 4><<<g, GAL_THREADS, 0, s>>>(fd, cd, rhop, vmask_f, Ttab32, kel32);
      if (nf) k_galerkin_fixed<float, 4><<<nf, 576, 0, s>>>(fd, cd, rhop, eactive_f, vmask_f, Ke, fixed_list, kel32);
    }
  } else {
    if (kel) {
      k_galerkin_gemm<double, 2><<<g, GAL_THREADS, 0, s>>>(fd, cd, rhop, vmask_f, Ttab64, kel);
      if (nf) k_galerkin_fixed<double, 2><<<nf, 576, 0, s>>>(fd, cd, rhop, eactive_f, vmask_f, Ke, fixed_list, kel);
    }
    if (kel32) {
      k_galerkin_gemm<float, 2><<<g, GAL_THREADS, 0, s>>>(fd, cd, rhop, vmask_f, Ttab32, kel32);
      if (nf) k_galerkin_fixed<float, 2><<<nf, 576, 0, s>>>(fd, cd, rhop, eactive_f, vmask_f, Ke, fixed_list, kel32);
    }
  }
}

template <typename T>
void launch_galerkin_dyadic_t(cudaStream_t s, const LevelDims& fd, const LevelDims& cd,
                              const uint8_t* eactive_f, const T* kel_f, T* kel_c) {
  k_galerkin_dyadic<T><<<(unsigned)cd.ne, 576, 0, s>>>(fd, cd, eactive_f, kel_f, kel_c);
}

template <typename T>
void launch_assemble_stencil_t(cudaStream_t s, const LevelDims& d, const uint8_t* eactive,
                               const uint8_t* vmask, const T* kel, T* st, T* planes) {
  k_assemble_stencil<T><<<nblk(27 * ((d.nv + 31) / 32 * 32), 256), 256, 0, s>>>(d, eactive, vmask, kel, st, st_idx<T>(d), planes);
}

void launch_stencil_planes(cudaStream_t s, const LevelDims& d, const double* st, double* planes) {
  k_stencil_planes<<<nblk(243 * d.nv, 256), 256, 0, s>>>(d.nv, st, st_idx<double>(d), planes);
}

bool stencil_by_vertex(const LevelDims& d) { return d.nv < STENCIL_WARP_MAX_NV; }

// Whether k_gj_sweep inverts a matrix of n unknowns (df_update: from FP32
// stencils) and, in blocks and smem, its launch: the triangle has to fit into the
// SMs' shared memory (n up to about 2,500).  Else, and for FP64 operators, the
// blocked Gauss-Jordan on A in place.
static bool coarsest_sweeps(int n, bool df_update, int nsm, int* blocks, size_t* smem) {
  const int64_t nt = (n + GJB - 1) / GJB, ntri = nt * (nt + 1) / 2;
  *blocks = nt == 1 ? 1 : (int)std::min<int64_t>(nsm, ntri + 1);
  const int64_t own = nt == 1 ? 1 : (ntri + *blocks - 2) / (*blocks - 1);
  *smem = (size_t)(8 * (4 * GJT + own * GJ_TILE));
  return df_update && *smem <= (size_t)GJ_SWEEP_SMEM;
}
static int sm_count() {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

// The matrix of the coarsest stencils; its symmetric part for the blocked form
// (the sweeps take that as they read).  Both here, before the inversion's stream
// starts: k_symmetrize in that stream let the set-up kernels of the design
// iteration onto the SMs first, and the blocked form's CTAs, two an SM, then came
// to lie unevenly (FP64 operators, 77x44x42: 18.8 against 15.0 ms an iteration).
template <typename T>
void launch_dense_from_stencil(cudaStream_t s, const LevelDims& d, const T* st, double* A) {
  const int64_t n = 3 * d.nv;
  cudaMemsetAsync(A, 0, sizeof(double) * n * n, s);
  k_dense_from_stencil<T><<<nblk(243 * d.nv, 256), 256, 0, s>>>(d, st, st_idx<T>(d), A);
  int blocks;
  size_t smem;
  if (!coarsest_sweeps((int)n, sizeof(T) == 4, sm_count(), &blocks, &smem))
    k_symmetrize<<<nblk(n * n, 256), 256, 0, s>>>((int)n, A);
}

// A: the coarsest matrix (launch_dense_from_stencil; its symmetric part is
// inverted in place), A32: the inverse in FP32.  max_per_sm: CTAs an SM of the
// blocked form.
int coarsest_invert(cudaStream_t s, int n, double* A, float* A32, double* work, int* status_dev, bool df_update,
                    int max_per_sm) {
  int blocks;
  size_t smem;
  const int nsm = sm_count();
  if (coarsest_sweeps(n, df_update, nsm, &blocks, &smem)) {
    static PerDeviceOnce once;
    const cudaError_t e = once_per_device(once, []() -> cudaError_t {
      return cudaFuncSetAttribute(k_gj_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, GJ_SWEEP_SMEM);
    });
    if (e != cudaSuccess) return (int)e;
    cudaMemsetAsync(status_dev, 0, 2 * sizeof(int), s);
    void* args[] = {&n, &A, &A32, &work, &status_dev};
    return (int)cudaLaunchCooperativeKernel((void*)k_gj_sweep, dim3(blocks), dim3(GJ_THREADS), args, smem, s);
  }
  const int threads = 256;
  int per_sm = 0;
  void* fn = df_update ? (void*)k_gj_blocked<true> : (void*)k_gj_blocked<false>;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0);
  if (per_sm < 1) return (int)cudaErrorCooperativeLaunchTooLarge;
  const int tiles = ((n + GJB - 1) / GJB) * ((n + GJB - 1) / GJB);
  blocks = std::max(1, std::min(tiles, nsm * std::min(per_sm, std::max(1, max_per_sm))));
  cudaMemsetAsync(status_dev, 0, 2 * sizeof(int), s);
  void* args[] = {&n, &A, &work, &status_dev};
  const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(threads), args, 0, s);
  if (e != cudaSuccess) return (int)e;
  launch_to_float(s, A, A32, (int64_t)n * n);
  return (int)cudaGetLastError();
}

void launch_to_float(cudaStream_t s, const double* a, float* b, int64_t n) {
  k_to_float<<<nblk(n, 256), 256, 0, s>>>(a, b, n);
}

template <typename T>
void launch_dense_gemv(cudaStream_t s, int n, const T* Ainv, const T* f_soa, T* u_soa, int64_t nv, int nb) {
  k_dense_gemv<T><<<dim3(nblk((int64_t)n * 32, 256), nb), 256, 0, s>>>(n, Ainv, f_soa, u_soa, nv);
}

template void launch_stencil_apply<double>(cudaStream_t, const LevelDims&, const double*, const double*,
                                           const double*, double*, bool, int);
template void launch_stencil_apply<float>(cudaStream_t, const LevelDims&, const float*, const float*,
                                          const float*, float*, bool, int);
template int launch_stencil_gs<double>(cudaStream_t, const LevelDims&, const double*, const uint8_t*,
                                       double*, const double*, int, bool);
template int launch_stencil_gs<float>(cudaStream_t, const LevelDims&, const float*, const uint8_t*,
                                      float*, const float*, int, bool);
template void launch_stencil_diag_inv<double>(cudaStream_t, const LevelDims&, const double*,
                                              const uint8_t*, double*);
template void launch_stencil_diag_inv<float>(cudaStream_t, const LevelDims&, const float*,
                                             const uint8_t*, float*);
template void launch_restrict<double>(cudaStream_t, const LevelDims&, const LevelDims&, const double*,
                                      double*, int);
template void launch_restrict<float>(cudaStream_t, const LevelDims&, const LevelDims&, const float*,
                                     float*, int);
template void launch_prolong<double>(cudaStream_t, const LevelDims&, const LevelDims&, const double*,
                                     double*, const uint8_t*, int);
template void launch_prolong<float>(cudaStream_t, const LevelDims&, const LevelDims&, const float*,
                                    float*, const uint8_t*, int);
template void launch_galerkin_dyadic_t<double>(cudaStream_t, const LevelDims&, const LevelDims&,
                                               const uint8_t*, const double*, double*);
template void launch_galerkin_dyadic_t<float>(cudaStream_t, const LevelDims&, const LevelDims&,
                                              const uint8_t*, const float*, float*);
template void launch_assemble_stencil_t<double>(cudaStream_t, const LevelDims&, const uint8_t*,
                                                const uint8_t*, const double*, double*, double*);
template void launch_assemble_stencil_t<float>(cudaStream_t, const LevelDims&, const uint8_t*,
                                               const uint8_t*, const float*, float*, float*);
template void launch_dense_from_stencil<double>(cudaStream_t, const LevelDims&, const double*, double*);
template void launch_dense_from_stencil<float>(cudaStream_t, const LevelDims&, const float*, double*);
template void launch_dense_gemv<double>(cudaStream_t, int, const double*, const double*, double*,
                                        int64_t, int);
template void launch_dense_gemv<float>(cudaStream_t, int, const float*, const float*, float*, int64_t, int);

}  // namespace topo
