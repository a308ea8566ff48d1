// Conjugate gradients with every search direction kept (internal to libsgpp_gb300): a step's direction
// is made conjugate to all the earlier ones instead of to the last alone, and a solve of the same
// operator with another right-hand side first takes its part in the span of the kept directions.
//
// Why: the operator's products are rounded (FP16 or FP32), so the two-term recurrence loses conjugacy to
// the directions of the large eigenvalues within some ten steps and finds them again and again, and a
// refinement that starts the next solve from nothing finds them once more. d = 10, level 5, 2^20 clustered
// points, to 1e-8: 90 steps of 0.92 ms; kept directions take 51 to 55 (the count of exact arithmetic).
//
// Cost: two passes over the kept vectors per step, 16 bytes per entry and direction, which the L2 holds
// at the grids' sizes (13,441 entries and 50 directions: 11 MB); both are spread over the chip, the dot
// products one block per direction (and piece of a long vector), the sums one block per 64 entries.
// Every sum has a fixed order.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_cluster.cuh"

namespace sgmev {

constexpr int kOrthoKept = 128;  // directions kept at most; then the last slot holds the latest one
constexpr int kOrthoThreads = 256;
constexpr int kOrthoEntries = 64;  // entries per block of ortho_apply_kernel, over 4 groups of directions
constexpr int kOrthoPieces = 16;   // pieces of a vector in ortho_dot_kernel, at most
constexpr int64_t kOrthoPiece = 16384;

// A solve's progress (squares): `mark`, the residual after the last step that took 30 % off it since the
// mark before, and `since`, the steps from there.
__host__ __device__ inline bool ortho_progress(double delta, double mark) { return delta < 0.5 * mark; }
// Whether a solve ends for want of it. Kept directions reach the floor that the products' rounding sets and
// creep from there (16 columns, d = 4 level 5, lambda 1e-5: 3,112 steps instead of 794 of the recurrence);
// once three digits are gained another refinement is the cheaper way on: 16 targets on d = 10 level 5, 2^20
// points, 26.5 / 30.9 / 33.7 fits/s after 32 / 16 / 8 such steps, at lambda 1e-7 268 / 265 / 297 ms (d = 6).
__host__ __device__ inline bool ortho_stands_still(int64_t since, double mark, double rhs) {
  return since >= (mark <= 1e-6 * rhs ? 16 : 128);
}
// Whether a fit goes on with the two-term recurrence (one direction kept, no standing still), as it always
// converges: a solve of 128 steps or more took less than a digit off the true residual (squares). Where far
// more steps are needed than directions are kept that can happen.
inline bool ortho_gives_up(int64_t steps, double before, double after) {
  return steps >= 128 && !(after <= 0.01 * before);
}

// pieces of a dot product of length n
inline int ortho_pieces(int64_t n) {
  const int64_t p = (n + kOrthoPiece - 1) / kOrthoPiece;
  return static_cast<int>(p < 1 ? 1 : p > kOrthoPieces ? kOrthoPieces : p);
}

// Vectors of `cols` independent columns, [np] each: direction j of column c at (j * cols + c) * np, its
// d.q at w[j * cols + c] (0: not one of the kept; its vectors are never read).

// part[(c * k + j) * pieces + s] = piece s of V_j . r in column c; grid (k directions, pieces, cols)
static __global__ void __launch_bounds__(kOrthoThreads)
    ortho_dot_kernel(int64_t n, int64_t np, const double* __restrict__ v, const double* __restrict__ w,
                     const double* __restrict__ r, double* __restrict__ part,
                     const double* __restrict__ stop) {
  if (*stop != 0.0) return;
  const int c = blockIdx.z, cols = gridDim.z, at = blockIdx.x * cols + c;
  if (w[at] == 0.0) return;
  __shared__ double sh[kOrthoThreads / 32];
  const int64_t len = (n + gridDim.y - 1) / gridDim.y;
  const int64_t a = blockIdx.y * len, b = a + len < n ? a + len : n;
  const double* vj = v + at * np;
  const double* rc = r + c * np;
  double acc = 0.0;
#pragma unroll 8
  for (int64_t i = a + threadIdx.x; i < b; i += kOrthoThreads) acc = fma(vj[i], rc[i], acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < kOrthoThreads / 32; ++i) s += sh[i];
    part[(static_cast<int64_t>(c) * gridDim.x + blockIdx.x) * gridDim.y + blockIdx.y] = s;
  }
}

// out = base + sign * sum_j (dot_j / w_j) V_j over k directions (base null: 0), zero beyond n; grid (entries,
// cols). out may be one of the V_j: a block has read its entries of all of them before it writes.
static __global__ void __launch_bounds__(kOrthoThreads)
    ortho_apply_kernel(int64_t n, int64_t np, int k, int pieces, const double* v, const double* __restrict__ w,
                       const double* __restrict__ part, double sign, const double* base, double* out,
                       const double* __restrict__ stop) {
  if (*stop != 0.0) return;
  constexpr int kGroups = kOrthoThreads / kOrthoEntries;
  __shared__ double c[kOrthoKept];
  __shared__ double sum[kGroups][kOrthoEntries];
  const int col = blockIdx.y, cols = gridDim.y;
  for (int j = threadIdx.x; j < k; j += kOrthoThreads) {
    const double wj = w[j * cols + col];
    double s = 0.0;
    if (wj != 0.0) {
      for (int p = 0; p < pieces; ++p) s += part[(static_cast<int64_t>(col) * k + j) * pieces + p];
      s = sign * s / wj;
    }
    c[j] = s;
  }
  __syncthreads();
  const int e = threadIdx.x % kOrthoEntries, g = threadIdx.x / kOrthoEntries;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kOrthoEntries + e;
  const int64_t o = static_cast<int64_t>(col) * np + i;
  double acc = 0.0;
  if (i < n) {
#pragma unroll 8
    for (int j = g; j < k; j += kGroups)
      if (c[j] != 0.0) acc = fma(c[j], v[static_cast<int64_t>(j) * cols * np + o], acc);
  }
  sum[g][e] = acc;
  __syncthreads();
  if (g == 0 && i < np) {
    double s = base && i < n ? base[o] : 0.0;
#pragma unroll
    for (int p = 0; p < kGroups; ++p) s += sum[p][e];
    out[o] = s;
  }
}

// A column's step along d (q = A d) on one cluster: where `take`, x += alpha d and r -= alpha q with
// alpha = r.d / d.q (nothing for d.q = 0); dq = d.q, rr = r.r
__device__ __forceinline__ void ortho_column_step(int64_t n, const double* __restrict__ d,
                                                  const double* __restrict__ q, double* __restrict__ x,
                                                  double* __restrict__ r, bool take, CgShared& sh,
                                                  double* dq_out, double* rr_out) {
  double adq = 0.0, ard = 0.0;
  for (int64_t i = cg_first(); i < n; i += kCgStride) {
    adq = fma(d[i], q[i], adq);
    ard = fma(r[i], d[i], ard);
  }
  const double dq = cg_cluster_sum(adq, sh, 0), rd = cg_cluster_sum(ard, sh, 1);
  take = take && dq != 0.0;
  const double alpha = take ? rd / dq : 0.0;
  double acc = 0.0;
  for (int64_t i = cg_first(); i < n; i += kCgStride) {
    double ri = r[i];
    if (take) {
      x[i] = fma(alpha, d[i], x[i]);
      ri = fma(-alpha, q[i], ri);
      r[i] = ri;
    }
    acc = fma(ri, ri, acc);
  }
  *dq_out = dq;
  *rr_out = cg_cluster_sum(acc, sh, 2);
}

// The step of one column: *w = d.q, scal[5] = the solve stops after this step, and {r.r, d.q} into
// page-locked memory. A step enqueued ahead of a stop does nothing.
static __global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kCgThreads)
    ortho_step_kernel(int64_t n, const double* __restrict__ d, const double* __restrict__ q,
                      double* __restrict__ x, double* __restrict__ r, double* __restrict__ scal,
                      double* __restrict__ w, double delta_0, double* __restrict__ host) {
  if (scal[5] != 0.0) return;
  __shared__ CgShared sh;
  double dq, rr;
  ortho_column_step(n, d, q, x, r, true, sh, &dq, &rr);
  cg_cluster_end();  // every block has read the stop flag and this block's sums
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *w = dq;
    scal[5] = dq == 0.0 || !(rr > delta_0) || !(rr > 0.0) ? 1.0 : 0.0;
    volatile double* h = host;
    h[0] = rr;
    h[1] = dq;
  }
}

// A step and the direction after it for short vectors, all in the cluster: block b holds entries
// [b len, (b+1) len) of r in shared memory, takes its part of the dot products with the k kept Q (this
// step's at `at` included), and forms its entries of the direction `next` from the cluster's sums. The
// three kernels that it replaces mostly start and wait: a whole iteration with 351 entries and 3,000 data
// points 55 -> 47 us, with 2,561 and 20,011 73 -> 67 us. Up to one entry a thread; above that the reads of
// the kept vectors are better spread over the chip.
constexpr int kOrthoShort = kCgCtas * kCgThreads;
static __global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kCgThreads)
    ortho_short_kernel(int n, int np, const double* p, const double* __restrict__ q,
                       double* __restrict__ w, int at, int k, double* next, double* __restrict__ x,
                       double* __restrict__ r, double* __restrict__ scal, double delta_0,
                       double* __restrict__ host) {
  namespace cg = cooperative_groups;
  if (scal[5] != 0.0) return;
  constexpr int kLen = kOrthoShort / kCgCtas;
  __shared__ CgShared sh;
  __shared__ double rs[kLen], dots[kOrthoKept], c[kOrthoKept];
  const int len = (n + kCgCtas - 1) / kCgCtas, b0 = static_cast<int>(blockIdx.x) * len;
  const int count = max(0, min(len, n - b0));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t own = static_cast<int64_t>(at) * np + b0;
  double dv = 0.0, qv = 0.0, rv = 0.0;  // len <= kCgThreads: an entry a thread
  if (tid < count) {
    dv = p[own + tid];
    qv = q[own + tid];
    rv = r[b0 + tid];
  }
  const double dq = cg_cluster_sum(dv * qv, sh, 0), rd = cg_cluster_sum(rv * dv, sh, 1);
  if (dq != 0.0 && tid < count) {
    const double alpha = rd / dq;
    x[b0 + tid] = fma(alpha, dv, x[b0 + tid]);
    rv = fma(-alpha, qv, rv);
    r[b0 + tid] = rv;
  }
  if (tid < count) rs[tid] = rv;
  __syncthreads();
  for (int j = warp; j < k; j += kCgThreads / 32) {
    const double* qj = q + static_cast<int64_t>(j) * np + b0;
    double acc = 0.0;
#pragma unroll 8
    for (int i = lane; i < count; i += 32) acc = fma(qj[i], rs[i], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) dots[j] = acc;
  }
  const double rr = cg_cluster_sum(rv * rv, sh, 2);  // (every block's dots are there after it)
  const bool stop = dq == 0.0 || !(rr > delta_0) || !(rr > 0.0);
  if (!stop) {
    if (tid < k) {
      double s = 0.0;
#pragma unroll
      for (int b = 0; b < kCgCtas; ++b) s += *cg::this_cluster().map_shared_rank(&dots[tid], b);
      c[tid] = s / (tid == at ? dq : w[tid]);
    }
    __syncthreads();
    if (tid < count) {
      double acc = 0.0;
#pragma unroll 8
      for (int j = 0; j < k; ++j) acc = fma(c[j], p[static_cast<int64_t>(j) * np + b0 + tid], acc);
      next[b0 + tid] = rv - acc;
    }
    if (blockIdx.x == kCgCtas - 1)
      for (int i = n + tid; i < np; i += kCgThreads) next[i] = 0.0;
  }
  cg_cluster_end();  // every block has read the stop flag and the others' sums
  if (blockIdx.x == 0 && tid == 0) {
    w[at] = dq;
    scal[5] = stop ? 1.0 : 0.0;
    volatile double* h = host;
    h[0] = rr;
    h[1] = dq;
  }
}

// out = base + sign * sum_j ((V_j . r) / w_j) U_j over the first k directions of `cols` columns, on
// stream s; v null: with the dot products of the call before. base null: 0.
inline cudaError_t ortho_combine(cudaStream_t s, int cols, int64_t n, int64_t np, int64_t k, const double* v,
                                 const double* r, const double* u, const double* w, double* part,
                                 double sign, const double* base, double* out, const double* stop) {
  const int pieces = ortho_pieces(n);
  if (v)
    ortho_dot_kernel<<<dim3(static_cast<unsigned>(k), static_cast<unsigned>(pieces),
                            static_cast<unsigned>(cols)),
                       kOrthoThreads, 0, s>>>(n, np, v, w, r, part, stop);
  ortho_apply_kernel<<<dim3(static_cast<unsigned>((np + kOrthoEntries - 1) / kOrthoEntries),
                            static_cast<unsigned>(cols)),
                       kOrthoThreads, 0, s>>>(n, np, static_cast<int>(k), pieces, u, w, part, sign,
                                              base, out, stop);
  return cudaGetLastError();
}

// directions that `bytes` hold of `cols` columns, between 2 (the two-term recurrence) and kOrthoKept
inline int64_t ortho_cap(int64_t bytes, int cols, int64_t np) {
  const int64_t c = bytes / (16 * cols * np);
  return c < 2 ? 2 : c > kOrthoKept ? kOrthoKept : c;
}

// doubles of the buffer for `cap` directions: P, Q, w and the dot products' pieces
inline size_t ortho_words(int64_t cap, int cols, int64_t np) {
  return static_cast<size_t>(cols) * static_cast<size_t>(cap) * (2 * static_cast<size_t>(np) + 1 + kOrthoPieces);
}

}  // namespace sgmev
