// Batched vector kernels of the multi-right-hand-side solver: nb vectors of
// length n stored one after another, one set of CG scalars per right-hand side.
// Reductions are deterministic: per-(CTA, rhs) partials that the right-hand
// side's last CTA adds in a fixed order.
#include <algorithm>

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
// CTA is last) and resets the counter.  part: [N][nb][gridDim.x].
template <int N>
__device__ __forceinline__ void bfinish(const double (&v)[N], double* part, double* const (&out)[N], unsigned* ctr) {
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
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double s = 0.0;
    for (int i = threadIdx.x; i < nblk; i += kThreads) s += __ldcg(part + ((int64_t)k * gridDim.y + rhs) * nblk + i);
    s = bsum(s);
    if (threadIdx.x == 0) out[k][rhs] = s;
  }
  if (threadIdx.x == 0) ctr[rhs] = 0u;
}

// a.b per right-hand side and, TWO, b.c with the same read of b.  The sums were
// finished by one thread a right-hand side, 256 dependent FP64 additions: 19 us
// after every 23 us of partial sums (eight vectors of 96x48x48).
template <typename T, bool TWO>
__global__ void __launch_bounds__(kThreads) k_bdot(const T* __restrict__ a, const T* __restrict__ b,
                                                   const T* __restrict__ c, int64_t n, double* __restrict__ part,
                                                   double* out0, double* out1, unsigned* ctr) {
  const int64_t off = (int64_t)blockIdx.y * n;
  double s = 0.0, t = 0.0;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    const double v = (double)b[off + i];
    s += (double)a[off + i] * v;
    if (TWO) t += v * (double)c[off + i];
  }
  if constexpr (TWO) {
    bfinish<2>({s, t}, part, {out0, out1}, ctr);
  } else {
    bfinish<1>({s}, part, {out0}, ctr);
  }
}

template <typename T>
void launch_bdot(cudaStream_t s, const T* a, const T* b, int64_t n, int nb, double* partial, unsigned* ctr, double* out,
                 const T* c, double* out_bc) {
  const dim3 g(bdot_blocks(n, nb), nb);
  if (c) k_bdot<T, true><<<g, kThreads, 0, s>>>(a, b, c, n, partial, out, out_bc, ctr);
  else k_bdot<T, false><<<g, kThreads, 0, s>>>(a, b, nullptr, n, partial, out, nullptr, ctr);
}
template void launch_bdot<double>(cudaStream_t, const double*, const double*, int64_t, int, double*, unsigned*, double*,
                                  const double*, double*);
template void launch_bdot<float>(cudaStream_t, const float*, const float*, int64_t, int, double*, unsigned*, double*,
                                 const float*, double*);

// Per right-hand side: beta = (rz - zrold) / rzold (first: 0).
__global__ void k_bbeta(int nb, const double* rz, const double* zrold, const double* rzold, int first, double* beta) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nb) return;
  beta[k] = first || !(rzold[k] != 0.0) ? 0.0 : (rz[k] - zrold[k]) / rzold[k];
}

// Per right-hand side: alpha = rz / dq while rr > rtol^2 ff, else 0 (the
// right-hand side has converged and its iterate is frozen); rzold = rz.
__global__ void k_balpha(int nb, const double* rz, const double* dq, const double* rr, const double* ff, double rtol2,
                         double* alpha, double* rzold) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nb) return;
  const bool active = rr[k] > rtol2 * ff[k] && dq[k] != 0.0;
  alpha[k] = active ? rz[k] / dq[k] : 0.0;
  rzold[k] = rz[k];
}

// d = z + beta d
template <typename T>
__global__ void k_bdir(int64_t n, int nb, const T* __restrict__ z, T* __restrict__ d, const double* __restrict__ beta) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * nb) return;
  const T b = (T)beta[i / n];
  d[i] = z[i] + b * d[i];
}

// x += alpha d, rold = r (when kept), r -= alpha q, and r.r of the new r
template <typename T>
__global__ void __launch_bounds__(kThreads) k_bupdate(int64_t n, T* __restrict__ x, T* __restrict__ r,
                                                      T* __restrict__ rold, const T* __restrict__ d,
                                                      const T* __restrict__ q, const double* __restrict__ alpha,
                                                      double* __restrict__ part, double* rr, unsigned* ctr) {
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
    s += (double)rn * (double)rn;
  }
  bfinish<1>({s}, part, {rr}, ctr);
}

void launch_bbeta(cudaStream_t s, int nb, const double* rz, const double* zrold, const double* rzold, bool first,
                  double* beta) {
  k_bbeta<<<nblk(nb, 64), 64, 0, s>>>(nb, rz, zrold, rzold, first ? 1 : 0, beta);
}
void launch_balpha(cudaStream_t s, int nb, const double* rz, const double* dq, const double* rr, const double* ff,
                   double rtol2, double* alpha, double* rzold) {
  k_balpha<<<nblk(nb, 64), 64, 0, s>>>(nb, rz, dq, rr, ff, rtol2, alpha, rzold);
}
template <typename T>
void launch_bdir(cudaStream_t s, int64_t n, int nb, const T* z, T* d, const double* beta) {
  k_bdir<T><<<nblk(n * nb, kThreads), kThreads, 0, s>>>(n, nb, z, d, beta);
}
template <typename T>
void launch_bupdate(cudaStream_t s, int64_t n, int nb, T* x, T* r, T* rold, const T* d, const T* q,
                    const double* alpha, double* partial, unsigned* ctr, double* rr) {
  k_bupdate<T><<<dim3(bdot_blocks(n, nb), nb), kThreads, 0, s>>>(n, x, r, rold, d, q, alpha, partial, rr, ctr);
}
template void launch_bdir<double>(cudaStream_t, int64_t, int, const double*, double*, const double*);
template void launch_bdir<float>(cudaStream_t, int64_t, int, const float*, float*, const double*);
template void launch_bupdate<double>(cudaStream_t, int64_t, int, double*, double*, double*, const double*,
                                     const double*, const double*, double*, unsigned*, double*);
template void launch_bupdate<float>(cudaStream_t, int64_t, int, float*, float*, float*, const float*, const float*,
                                    const double*, double*, unsigned*, double*);

}  // namespace topo
