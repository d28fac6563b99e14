// Vector kernels: deterministic two-pass FP64 reductions, axpy-type updates
// and the Chebyshev smoothing step.
#include <algorithm>

#include "topo_internal.h"

namespace topo {

constexpr int RED_THREADS = 256;

template <typename T, int W>
struct alignas(16) Pack16 {
  T v[W];
};
constexpr int RED_MAX_BLOCKS = 1024;

static inline unsigned nblk(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Four values a thread: with eight, vectors of a small level (100 k) were on
// too few SMs and waited for each value in turn.
int reduce_blocks(int64_t n) {
  int64_t b = (n + RED_THREADS * 4 - 1) / (RED_THREADS * 4);
  if (b < 1) b = 1;
  if (b > RED_MAX_BLOCKS) b = RED_MAX_BLOCKS;
  return (int)b;
}

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double ws[RED_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) ws[w] = v;
  __syncthreads();
  double s = 0.0;
  if (w == 0) {
    s = lane < RED_THREADS / 32 ? ws[lane] : 0.0;
#pragma unroll
    for (int o = RED_THREADS / 64; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  }
  return s;  // valid in thread 0
}

// Completion by the last block: each block's thread 0 has published its partial;
// every block then takes a ticket, and the block with the last one sums all nb
// partials in index order (the order of k_finalize_sum, so the result does not
// depend on which block finishes last) and resets the counter for the next use.
// Saves the separate finalising launch.  ctr: one counter per stream in order.
// One call sums K sets of partials, set k at partial + k nb, into *out[k] (null:
// not wanted) and tot[k]; true in thread 0 of the last block, which goes on from
// there.
template <int K>
__device__ __forceinline__ bool finish_sums(const double* partial, int nb, double* const (&out)[K], double (&tot)[K],
                                            unsigned* ctr) {
  __shared__ bool last;
  if (threadIdx.x == 0) last = last_ticket(ctr, (unsigned)nb);  // thread 0 wrote the block's partials
  __syncthreads();
  if (!last) return false;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    tot[k] = 0.0;
    if (!out[k]) continue;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) tot[k] += __ldcg(partial + (int64_t)k * nb + i);
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (!out[k]) continue;
    if (k > 0) __syncthreads();  // block_sum's shared words are free again
    tot[k] = block_sum(tot[k]);
    if (threadIdx.x == 0) *out[k] = tot[k];
  }
  if (threadIdx.x == 0) *ctr = 0u;
  return threadIdx.x == 0;
}

// Per-thread partial sums are accumulated in the vector's precision (FP32
// vectors: a few dozen terms per thread, inside the FP32 inner solver only) and
// combined in FP64 across threads and blocks.  With ctr the last block also
// writes the total to out, and the ratio after it.
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_dot_partial(const T* __restrict__ a, const T* __restrict__ b,
                                                             int64_t n, double* __restrict__ partial,
                                                             double* __restrict__ out = nullptr,
                                                             unsigned* __restrict__ ctr = nullptr,
                                                             SumRatio rt = SumRatio{}) {
  T s = T(0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += a[i] * (b ? b[i] : T(1));
  const double bs = block_sum((double)s);
  if (threadIdx.x == 0) partial[blockIdx.x] = bs;
  if (ctr) {
    double* const outs[1] = {out};
    double tot[1];
    RatioOps ops{};
    if (threadIdx.x == 0) ops = ratio_load(rt);
    if (finish_sums(partial, gridDim.x, outs, tot, ctr)) ratio_write(rt, ops, out, tot[0]);
  }
}

// The flexible CG's r.z and z.rold (a.b and b.c) with one read of z and one
// launch: k_dot_partial's sums in the same order.  The FP64 vectors of an outer
// step are read once less (n = 92 k: 2 x 7.9 us -> one launch).
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_dot2(const T* __restrict__ a, const T* __restrict__ b,
                                                      const T* __restrict__ c, int64_t n,
                                                      double* __restrict__ partial, double* out_ab, double* out_bc,
                                                      unsigned* __restrict__ ctr,
                                                      const double* __restrict__ skip_if_zero, SumRatio rt) {
  const bool two = !(skip_if_zero && *skip_if_zero == 0.0);  // the same in every thread of the grid
  T s = T(0), t = T(0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T bi = b[i];
    s += a[i] * bi;
    if (two) t += bi * c[i];
  }
  const double bs = block_sum((double)s);
  if (threadIdx.x == 0) partial[blockIdx.x] = bs;
  if (two) {
    __syncthreads();  // block_sum's shared words are free again
    const double bt = block_sum((double)t);
    if (threadIdx.x == 0) partial[gridDim.x + blockIdx.x] = bt;
  }
  double* const outs[2] = {out_ab, two ? out_bc : nullptr};
  double tot[2];
  RatioOps ops{};
  if (threadIdx.x == 0) ops = ratio_load(rt);
  if (finish_sums(partial, gridDim.x, outs, tot, ctr) && two) ratio_write(rt, ops, out_ab, tot[0], out_bc, tot[1]);
}

__global__ void __launch_bounds__(RED_THREADS) k_finalize_sum(const double* __restrict__ partial, int nb, double* out,
                                                              SumRatio rt) {
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) s += partial[i];
  s = block_sum(s);
  if (threadIdx.x == 0) {
    *out = s;
    ratio_write(rt, ratio_load(rt), out, s);
  }
}

__global__ void __launch_bounds__(RED_THREADS) k_maxabs_partial(const double* __restrict__ a, int64_t n,
                                                                double* __restrict__ partial) {
  double m = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = fmax(m, fabs(a[i]));
  __shared__ double ws[RED_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int w = 0; w < RED_THREADS / 32; ++w) r = fmax(r, ws[w]);
    partial[blockIdx.x] = r;
  }
}

__global__ void k_finalize_max(const double* __restrict__ partial, int nb, double* __restrict__ out) {
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int i = 0; i < nb; ++i) r = fmax(r, partial[i]);
    *out = r;
  }
}

template <typename T>
void launch_dot(cudaStream_t s, const T* a, const T* b, int64_t n, double* partial, double* out, unsigned* ctr,
                SumRatio rt) {
  const int nb = reduce_blocks(n);
  if (ctr) {
    k_dot_partial<T><<<nb, RED_THREADS, 0, s>>>(a, b, n, partial, out, ctr, rt);
  } else {
    k_dot_partial<T><<<nb, RED_THREADS, 0, s>>>(a, b, n, partial);
    k_finalize_sum<<<1, RED_THREADS, 0, s>>>(partial, nb, out, rt);
  }
}

template <typename T>
void launch_dot2(cudaStream_t s, const T* a, const T* b, const T* c, int64_t n, double* partial, double* out_ab,
                 double* out_bc, unsigned* ctr, const double* skip_if_zero, SumRatio rt) {
  k_dot2<T><<<reduce_blocks(n), RED_THREADS, 0, s>>>(a, b, c, n, partial, out_ab, out_bc, ctr, skip_if_zero, rt);
}

void launch_sum_partials(cudaStream_t s, const double* partial, int nb, double* out, SumRatio rt) {
  k_finalize_sum<<<1, RED_THREADS, 0, s>>>(partial, nb, out, rt);
}

void launch_sum(cudaStream_t s, const double* a, int64_t n, double* partial, double* out) {
  const int nb = reduce_blocks(n);
  k_dot_partial<double><<<nb, RED_THREADS, 0, s>>>(a, nullptr, n, partial);
  k_finalize_sum<<<1, RED_THREADS, 0, s>>>(partial, nb, out, SumRatio{});
}

void launch_maxabs(cudaStream_t s, const double* a, int64_t n, double* partial, double* out) {
  const int nb = reduce_blocks(n);
  k_maxabs_partial<<<nb, RED_THREADS, 0, s>>>(a, n, partial);
  k_finalize_max<<<1, 32, 0, s>>>(partial, nb, out);
}

__global__ void k_axpby(double a, const double* __restrict__ x, double b, double* __restrict__ y, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = a * x[i] + b * y[i];
}

void launch_axpby(cudaStream_t s, double a, const double* x, double b, double* y, int64_t n) {
  k_axpby<<<nblk(n, 256), 256, 0, s>>>(a, x, b, y, n);
}

template <typename T>
__global__ void k_fill(T* a, T v, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

template <typename T>
void launch_fill(cudaStream_t s, T* a, T v, int64_t n) {
  k_fill<T><<<nblk(n, 256), 256, 0, s>>>(a, v, n);
}

template <typename T>
void launch_copy(cudaStream_t s, const T* a, T* b, int64_t n) {
  cudaMemcpyAsync(b, a, sizeof(T) * n, cudaMemcpyDeviceToDevice, s);
}

__global__ void k_d2f(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}
__global__ void k_f2d_add(const float* __restrict__ a, double* __restrict__ b, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] += (double)a[i];
}
void launch_d2f(cudaStream_t s, const double* a, float* b, int64_t n) {
  k_d2f<<<nblk(n, 256), 256, 0, s>>>(a, b, n);
}
void launch_f2d_add(cudaStream_t s, const float* a, double* b, int64_t n) {
  k_f2d_add<<<nblk(n, 256), 256, 0, s>>>(a, b, n);
}

// d = z + beta d (beta = sc[beta_slot]), or d = z.  With first_if_zero the
// choice is made on the device: d = z when *first_if_zero is 0 (an iteration
// counter).
template <typename T>
__global__ void k_pcg_dir(const T* __restrict__ z, T* __restrict__ d, const double* __restrict__ sc,
                          int beta_slot, bool first_host, int64_t n, int packed,
                          const double* __restrict__ first_if_zero) {
  constexpr int W = 16 / sizeof(T);
  using P = Pack16<T, W>;
  const bool first = first_if_zero ? (*first_if_zero == 0.0) : first_host;
  const T beta = first ? T(0) : (T)sc[beta_slot];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t npk = packed ? n / W : 0;
  if (i < npk) {
    const P zp = reinterpret_cast<const P*>(z)[i];
    P dp = first ? zp : reinterpret_cast<const P*>(d)[i];
    if (!first) {
#pragma unroll
      for (int k = 0; k < W; ++k) dp.v[k] = zp.v[k] + beta * dp.v[k];
    }
    reinterpret_cast<P*>(d)[i] = dp;
  }
  // scalar elements: the tail past the last pack, or all of them unpacked
  const int64_t j = packed ? npk * W + i : i;
  if ((!packed || i < W) && j < n) d[j] = first ? z[j] : z[j] + beta * d[j];
}

// d = z (first) or z + beta d, in 16-byte packs when both vectors are aligned
template <typename T>
void launch_pcg_dir(cudaStream_t s, const T* z, T* d, const double* sc, int beta_slot, bool first,
                    int64_t n, const double* first_if_zero) {
  constexpr int W = 16 / sizeof(T);
  const bool packed = (((uintptr_t)z | (uintptr_t)d) & 15) == 0;
  const int64_t threads = packed ? std::max<int64_t>(n / W, W) : n;
  k_pcg_dir<T><<<nblk(threads, 256), 256, 0, s>>>(z, d, sc, beta_slot, first, n, packed ? 1 : 0, first_if_zero);
}

// x += alpha d, rold = r, r -= alpha q (alpha = sc[alpha_slot]), fused with the
// new residual's squared norm: per-thread sums
// in the vectors' precision, combined in FP64 in a fixed order (deterministic).
// Each thread moves 16-byte packs (4 floats / 2 doubles) so enough bytes are in
// flight to stream at HBM bandwidth; the tail past the last whole pack is scalar.
// FP64 has two packs of each vector in flight at four CTAs an SM (64 registers):
// 256x128x128 148 -> 110 us (6.5 TB/s), 159x79x77 34.8 -> 33.1 us; without the bound
// 122 and 41 us.
// The last block also closes the iteration (the r.z kept for the next beta, the
// device loop's count and test): every block has read alpha by then, and a
// copy node and a one-thread kernel are saved per iteration.
template <typename T>
__global__ void __launch_bounds__(RED_THREADS, sizeof(T) == 8 ? 4 : 0) k_pcg_update_rr(T* __restrict__ x, T* __restrict__ r,
                                                               T* __restrict__ rold, const T* __restrict__ d,
                                                               const T* __restrict__ q, double* sc, int alpha_slot,
                                                               int rz_slot, int rzold_slot, int64_t n,
                                                               double* __restrict__ partial, int packed, double* rr,
                                                               unsigned* __restrict__ ctr, LoopCtl lc) {
  constexpr int W = 16 / sizeof(T);
  using P = Pack16<T, W>;
  const T alpha = (T)sc[alpha_slot];
  T acc = T(0);
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gs = (int64_t)gridDim.x * blockDim.x;
  const int64_t npk = packed ? n / W : 0;
  auto step = [&](int64_t i, const P& rp, const P& xp, const P& dp, const P& qp) {
    P xn, rn;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      xn.v[k] = xp.v[k] + alpha * dp.v[k];
      rn.v[k] = rp.v[k] - alpha * qp.v[k];
      acc += rn.v[k] * rn.v[k];
    }
    if (rold) reinterpret_cast<P*>(rold)[i] = rp;
    reinterpret_cast<P*>(x)[i] = xn;
    reinterpret_cast<P*>(r)[i] = rn;
  };
  int64_t i0 = gid;
  if constexpr (sizeof(T) == 8) {  // two packs of each vector asked for before the first is used
    for (; i0 + gs < npk; i0 += 2 * gs) {
      P rp[2], xp[2], dp[2], qp[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int64_t i = i0 + j * gs;
        rp[j] = reinterpret_cast<const P*>(r)[i];
        xp[j] = reinterpret_cast<const P*>(x)[i];
        dp[j] = reinterpret_cast<const P*>(d)[i];
        qp[j] = reinterpret_cast<const P*>(q)[i];
      }
      step(i0, rp[0], xp[0], dp[0], qp[0]);
      step(i0 + gs, rp[1], xp[1], dp[1], qp[1]);
    }
  }
  for (int64_t i = i0; i < npk; i += gs) {
    const P rp = reinterpret_cast<const P*>(r)[i], xp = reinterpret_cast<const P*>(x)[i];
    const P dp = reinterpret_cast<const P*>(d)[i], qp = reinterpret_cast<const P*>(q)[i];
    step(i, rp, xp, dp, qp);
  }
  for (int64_t i = npk * W + gid; i < n; i += gs) {
    const T ri = r[i];
    if (rold) rold[i] = ri;
    x[i] = x[i] + alpha * d[i];
    const T rn = ri - alpha * q[i];
    r[i] = rn;
    acc += rn * rn;
  }
  const double bs = block_sum((double)acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = bs;
  double* const outs[1] = {rr};
  double tot[1], rz = 0.0;
  LoopSlots ls{};
  if (threadIdx.x == 0) {
    rz = __ldcg(sc + rz_slot);
    ls = loop_load(lc);
  }
  if (finish_sums(partial, gridDim.x, outs, tot, ctr)) {
    sc[rzold_slot] = rz;
    if (lc.loop) loop_step(lc, ls, tot[0]);
  }
}

template <typename T>
void launch_pcg_update_rr(cudaStream_t s, T* x, T* r, T* rold, const T* d, const T* q, double* sc,
                          int alpha_slot, int rz_slot, int rzold_slot, int64_t n, double* partial, double* rr,
                          unsigned* ctr, LoopCtl lc) {
  // 16-byte packs when all five vectors start on 16-byte boundaries
  const uintptr_t al = (uintptr_t)x | (uintptr_t)r | (uintptr_t)rold | (uintptr_t)d | (uintptr_t)q;
  const int nb = reduce_blocks(n);
  k_pcg_update_rr<T><<<nb, RED_THREADS, 0, s>>>(x, r, rold, d, q, sc, alpha_slot, rz_slot, rzold_slot, n, partial,
                                                 (al & 15) == 0, rr, ctr, lc);
}

// Start of an inner CG: the FP64 residual rounded to FP32, x = 0, the rounded
// residual's squared norm (k_dot_partial's sum, term by term) and the loop's
// start in one pass instead of a conversion, a fill, a dot and a one-thread
// kernel that each wait for the one before (4 launches of 1.4 us and more per
// outer step; the vector is read once instead of twice).
__global__ void __launch_bounds__(RED_THREADS) k_inner_start(const double* __restrict__ r, float* __restrict__ r32,
                                                             float* __restrict__ x32, int64_t n,
                                                             double* __restrict__ partial, double* rr,
                                                             const double* bb, unsigned* __restrict__ ctr,
                                                             LoopCtl lc) {
  float s = 0.f;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = (float)r[i];
    r32[i] = v;
    x32[i] = 0.f;
    s += v * v;
  }
  const double bs = block_sum((double)s);
  if (threadIdx.x == 0) partial[blockIdx.x] = bs;
  double* const outs[1] = {rr};
  double tot[1];
  const double b2 = threadIdx.x == 0 ? __ldcg(bb) : 0.0;
  if (finish_sums(partial, gridDim.x, outs, tot, ctr)) loop_start(lc, b2, tot[0]);
}

void launch_inner_start(cudaStream_t s, const double* r, float* r32, float* x32, int64_t n, double* partial,
                        double* rr, const double* bb, unsigned* ctr, LoopCtl lc) {
  k_inner_start<<<reduce_blocks(n), RED_THREADS, 0, s>>>(r, r32, x32, n, partial, rr, bb, ctr, lc);
}

// A power step after the operator: the block inverse, the normalisation of x
// (applied here, the operator being linear) and both sums the step needs, x.z
// for the Rayleigh estimate and z.z for the next normalisation.  The blocks
// take the old norm before their ticket, so the last one may replace it.  Two
// launches a step (with the operator) instead of four: at small levels each
// one is a launch and a wait of 3 to 8 us for a few KB of vectors.  As many
// blocks as vertices fill, up to the reduction's bound (a block's FP64 sums
// cost more than the loop's own work beyond that).
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_power_step(int64_t nv, const T* __restrict__ dinv, bool sym,
                                                            const T* __restrict__ x, const T* __restrict__ y,
                                                            T* __restrict__ z, double* __restrict__ partial,
                                                            double* nrm, double* xx, double* xz,
                                                            unsigned* __restrict__ ctr) {
  const double n2 = *nrm;
  const T sc = (T)rsqrt(n2);
  T sxz = T(0), szz = T(0);
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
    const T r0 = y[v] * sc, r1 = y[nv + v] * sc, r2 = y[2 * nv + v] * sc;
    T z0, z1, z2;
    bool done = false;
    if constexpr (sizeof(T) == 4) {
      if (sym) {
        const float4 a = reinterpret_cast<const float4*>(dinv)[v];
        const float2 b = reinterpret_cast<const float2*>(dinv + 4 * nv)[v];
        z0 = a.x * r0 + a.y * r1 + a.z * r2;
        z1 = a.y * r0 + a.w * r1 + b.x * r2;
        z2 = a.z * r0 + b.x * r1 + b.y * r2;
        done = true;
      }
    }
    if (!done) {
      z0 = dinv[v] * r0 + dinv[nv + v] * r1 + dinv[2 * nv + v] * r2;
      z1 = dinv[3 * nv + v] * r0 + dinv[4 * nv + v] * r1 + dinv[5 * nv + v] * r2;
      z2 = dinv[6 * nv + v] * r0 + dinv[7 * nv + v] * r1 + dinv[8 * nv + v] * r2;
    }
    sxz += x[v] * z0 + x[nv + v] * z1 + x[2 * nv + v] * z2;
    szz += z0 * z0 + z1 * z1 + z2 * z2;
    z[v] = z0;
    z[nv + v] = z1;
    z[2 * nv + v] = z2;
  }
  const double b0 = block_sum((double)sxz);
  if (threadIdx.x == 0) partial[blockIdx.x] = b0;
  __syncthreads();  // block_sum's shared words are free again
  const double b1 = block_sum((double)szz);
  if (threadIdx.x == 0) partial[gridDim.x + blockIdx.x] = b1;
  double* const outs[2] = {xz, nrm};
  double tot[2];
  if (finish_sums(partial, gridDim.x, outs, tot, ctr)) *xx = n2;
}

template <typename T>
void launch_power_step(cudaStream_t s, int64_t nv, const T* dinv, bool sym, const T* x, const T* y, T* z,
                       double* partial, double* nrm, double* xx, double* xz, unsigned* ctr) {
  const int nb = (int)std::min<int64_t>(nblk(nv, RED_THREADS), RED_MAX_BLOCKS);
  k_power_step<T><<<nb, RED_THREADS, 0, s>>>(nv, dinv, sym, x, y, z, partial, nrm, xx, xz, ctr);
}

template void launch_pcg_update_rr<double>(cudaStream_t, double*, double*, double*, const double*, const double*,
                                           double*, int, int, int, int64_t, double*, double*, unsigned*, LoopCtl);
template void launch_pcg_update_rr<float>(cudaStream_t, float*, float*, float*, const float*, const float*,
                                          double*, int, int, int, int64_t, double*, double*, unsigned*, LoopCtl);
template void launch_power_step<double>(cudaStream_t, int64_t, const double*, bool, const double*, const double*,
                                        double*, double*, double*, double*, double*, unsigned*);
template void launch_power_step<float>(cudaStream_t, int64_t, const float*, bool, const float*, const float*, float*,
                                       double*, double*, double*, double*, unsigned*);
template void launch_dot<double>(cudaStream_t, const double*, const double*, int64_t, double*, double*, unsigned*,
                                  SumRatio);
template void launch_dot<float>(cudaStream_t, const float*, const float*, int64_t, double*, double*, unsigned*,
                                 SumRatio);
template void launch_dot2<double>(cudaStream_t, const double*, const double*, const double*, int64_t, double*, double*,
                                  double*, unsigned*, const double*, SumRatio);
template void launch_dot2<float>(cudaStream_t, const float*, const float*, const float*, int64_t, double*, double*,
                                 double*, unsigned*, const double*, SumRatio);
template void launch_fill<double>(cudaStream_t, double*, double, int64_t);
template void launch_fill<float>(cudaStream_t, float*, float, int64_t);
template void launch_copy<double>(cudaStream_t, const double*, double*, int64_t);
template void launch_copy<float>(cudaStream_t, const float*, float*, int64_t);
template void launch_pcg_dir<double>(cudaStream_t, const double*, double*, const double*, int, bool, int64_t,
                                      const double*);
template void launch_pcg_dir<float>(cudaStream_t, const float*, float*, const double*, int, bool, int64_t,
                                     const double*);

}  // namespace topo
