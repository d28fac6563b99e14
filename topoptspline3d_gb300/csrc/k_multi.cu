// Batched vector kernels of the multi-right-hand-side solver: nb vectors of
// length n stored one after another, one set of CG scalars per right-hand side.
// Reductions are deterministic: per-(CTA, rhs) partials that the right-hand
// side's last CTA adds in a fixed order.
#include <algorithm>
#include <type_traits>

#include "topo_internal.h"

namespace topo {

namespace {
constexpr int kThreads = 256;
inline unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }
}  // namespace

// CTAs per right-hand side of the reductions: eight CTAs an SM over the batch,
// at most kMaxBlocks (the partials' room).
constexpr int kMaxBlocks = 256;
inline int bdot_blocks(int64_t n, int nb) {
  const int64_t fill = (152 * 8 + nb - 1) / nb;
  return (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)kMaxBlocks, fill, (n + kThreads - 1) / kThreads}));
}

// Sum of v over the CTA, valid in thread 0.
__device__ __forceinline__ double bsum(double v) {
  __shared__ double ws[kThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) ws[w] = v;
  __syncthreads();
  double s = 0.0;
  if (w == 0) {
    s = lane < kThreads / 32 ? ws[lane] : 0.0;
#pragma unroll
    for (int o = kThreads / 64; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  }
  return s;
}

// Publishes the CTA's sums; the CTA that takes the right-hand side's last
// ticket adds its partials in index order (the result does not depend on which
// CTA is last), resets the counter and calls fin with the totals in one thread.
// part: [N][nb][gridDim.x].
template <int N, typename Fin>
__device__ __forceinline__ void bfinish(const double (&v)[N], double* part, unsigned* ctr, Fin&& fin) {
  __shared__ bool last;
  const int rhs = blockIdx.y, nblk = gridDim.x;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double s = bsum(v[k]);
    if (threadIdx.x == 0) part[((int64_t)k * gridDim.y + rhs) * nblk + blockIdx.x] = s;
  }
  if (threadIdx.x == 0) last = last_ticket(ctr + rhs, (unsigned)nblk);
  __syncthreads();
  if (!last) return;
  double tot[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    tot[k] = 0.0;
    for (int i = threadIdx.x; i < nblk; i += kThreads) tot[k] += __ldcg(part + ((int64_t)k * gridDim.y + rhs) * nblk + i);
  }
#pragma unroll
  for (int k = 0; k < N; ++k) tot[k] = bsum(tot[k]);
  if (threadIdx.x == 0) {
    ctr[rhs] = 0u;
    fin(tot);
  }
}

// What a dot is followed by, per right-hand side, in the thread that has its
// total (a kernel of its own took 3 to 4 us a scalar).
struct BNone {};
// beta = (rz - zrold) / rzold (0 at first, and for a right-hand side of rzold = 0)
struct BBeta {
  const double* rzold;
  double* beta;
  int first;
};
// alpha = rz / dq while rr > rtol^2 ff, else 0 (the right-hand side has
// converged and its iterate is frozen); rzold = rz
struct BAlpha {
  const double *rz, *rr, *ff;
  double rtol2;
  double *alpha, *rzold;
};

// out = a.b per right-hand side, and the step St; TWO: with b.c by the same read
// of b, for beta.  b may be of the other precision (the preconditioner's FP32
// result in the FP64 iteration: widening it in memory first cost a pass of 12
// bytes a value and twice the reads here).  Bound: two FP64 lanes a clock and SM
// against 8 to 20 bytes a value, so four values are in flight a thread.
template <typename T, typename TB, bool TWO, typename St>
__global__ void __launch_bounds__(kThreads) k_bdot(const T* __restrict__ a, const TB* __restrict__ b,
                                                   const T* __restrict__ c, int64_t n, double* __restrict__ part,
                                                   double* out, unsigned* ctr, St st) {
  const int rhs = blockIdx.y;
  const int64_t off = (int64_t)rhs * n;
  double w0 = 0.0, w1 = 0.0, w2 = 0.0;  // the step's operands, read ahead
  if constexpr (std::is_same<St, BBeta>::value) {
    w0 = st.rzold[rhs];
  } else if constexpr (std::is_same<St, BAlpha>::value) {
    w0 = st.rz[rhs];
    w1 = st.rr[rhs];
    w2 = st.ff[rhs];
  }
  double s = 0.0, t = 0.0;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    const double v = (double)b[off + i];
    s += (double)a[off + i] * v;
    if (TWO) t += v * (double)c[off + i];
  }
  auto fin = [&](double ab, double bc) {
    out[rhs] = ab;
    if constexpr (std::is_same<St, BBeta>::value) {
      st.beta[rhs] = st.first || !(w0 != 0.0) ? 0.0 : (ab - bc) / w0;
    } else if constexpr (std::is_same<St, BAlpha>::value) {
      st.alpha[rhs] = w1 > st.rtol2 * w2 && ab != 0.0 ? w0 / ab : 0.0;
      st.rzold[rhs] = w0;
    }
  };
  if constexpr (TWO) bfinish<2>({s, t}, part, ctr, [&](const double(&q)[2]) { fin(q[0], q[1]); });
  else bfinish<1>({s}, part, ctr, [&](const double(&q)[1]) { fin(q[0], 0.0); });
}

template <typename T>
void launch_bdot(cudaStream_t s, const T* a, const T* b, int64_t n, int nb, double* partial, unsigned* ctr,
                 double* out) {
  k_bdot<T, T, false, BNone><<<dim3(bdot_blocks(n, nb), nb), kThreads, 0, s>>>(a, b, nullptr, n, partial, out, ctr,
                                                                              BNone{});
}
template <typename T>
void launch_bdot_beta(cudaStream_t s, const T* r, const float* z, const T* rold, int64_t n, int nb, double* partial,
                      unsigned* ctr, double* rz, const double* rzold, bool first, double* beta) {
  const dim3 g(bdot_blocks(n, nb), nb);
  const BBeta st{rzold, beta, first ? 1 : 0};
  if (rold) k_bdot<T, float, true, BBeta><<<g, kThreads, 0, s>>>(r, z, rold, n, partial, rz, ctr, st);
  else k_bdot<T, float, false, BBeta><<<g, kThreads, 0, s>>>(r, z, nullptr, n, partial, rz, ctr, st);
}
template <typename T>
void launch_bdot_alpha(cudaStream_t s, const T* d, const T* q, int64_t n, int nb, double* partial, unsigned* ctr,
                       double* dq, const double* rz, const double* rr, const double* ff, double rtol2, double* alpha,
                       double* rzold) {
  k_bdot<T, T, false, BAlpha><<<dim3(bdot_blocks(n, nb), nb), kThreads, 0, s>>>(
      d, q, nullptr, n, partial, dq, ctr, BAlpha{rz, rr, ff, rtol2, alpha, rzold});
}

// d = z + beta d, z in FP32
constexpr int kDirEach = 4;  // values of a thread, in flight together
template <typename T>
__global__ void __launch_bounds__(kThreads) k_bdir(int64_t n, const float* __restrict__ z, T* __restrict__ d,
                                                   const double* __restrict__ beta) {
  const int64_t off = (int64_t)blockIdx.y * n, i0 = (int64_t)blockIdx.x * (kDirEach * kThreads) + threadIdx.x;
  const T b = (T)beta[blockIdx.y];
#pragma unroll
  for (int k = 0; k < kDirEach; ++k) {
    const int64_t i = i0 + k * kThreads;
    if (i < n) d[off + i] = (T)z[off + i] + b * d[off + i];
  }
}

// x += alpha d, rold = r (when kept), r -= alpha q, r.r of the new r, and the
// new r in FP32 for the preconditioner (when wanted: it is in registers here)
template <typename T>
__global__ void __launch_bounds__(kThreads) k_bupdate(int64_t n, T* __restrict__ x, T* __restrict__ r,
                                                      T* __restrict__ rold, float* __restrict__ r32,
                                                      const T* __restrict__ d, const T* __restrict__ q,
                                                      const double* __restrict__ alpha, double* __restrict__ part,
                                                      double* rr, unsigned* ctr) {
  const int64_t off = (int64_t)blockIdx.y * n;
  const T a = (T)alpha[blockIdx.y];
  double s = 0.0;
#pragma unroll 2
  for (int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x; k < n; k += (int64_t)gridDim.x * kThreads) {
    const int64_t i = off + k;
    const T r0 = r[i];
    x[i] += a * d[i];
    if (rold) rold[i] = r0;
    const T rn = r0 - a * q[i];
    r[i] = rn;
    if (r32) r32[i] = (float)rn;
    s += (double)rn * (double)rn;
  }
  bfinish<1>({s}, part, ctr, [&](const double(&t)[1]) { rr[blockIdx.y] = t[0]; });
}

template <typename T>
void launch_bdir(cudaStream_t s, int64_t n, int nb, const float* z, T* d, const double* beta) {
  k_bdir<T><<<dim3(nblk(n, kDirEach * kThreads), nb), kThreads, 0, s>>>(n, z, d, beta);
}
template <typename T>
void launch_bupdate(cudaStream_t s, int64_t n, int nb, T* x, T* r, T* rold, float* r32, const T* d, const T* q,
                    const double* alpha, double* partial, unsigned* ctr, double* rr) {
  k_bupdate<T><<<dim3(bdot_blocks(n, nb), nb), kThreads, 0, s>>>(n, x, r, rold, r32, d, q, alpha, partial, rr, ctr);
}
#define TOPO_MULTI(T)                                                                                                  \
  template void launch_bdot<T>(cudaStream_t, const T*, const T*, int64_t, int, double*, unsigned*, double*);           \
  template void launch_bdot_beta<T>(cudaStream_t, const T*, const float*, const T*, int64_t, int, double*, unsigned*,  \
                                    double*, const double*, bool, double*);                                            \
  template void launch_bdot_alpha<T>(cudaStream_t, const T*, const T*, int64_t, int, double*, unsigned*, double*,      \
                                     const double*, const double*, const double*, double, double*, double*);           \
  template void launch_bdir<T>(cudaStream_t, int64_t, int, const float*, T*, const double*);                           \
  template void launch_bupdate<T>(cudaStream_t, int64_t, int, T*, T*, T*, float*, const T*, const T*, const double*,   \
                                  double*, unsigned*, double*);
TOPO_MULTI(double)
TOPO_MULTI(float)
#undef TOPO_MULTI

}  // namespace topo
