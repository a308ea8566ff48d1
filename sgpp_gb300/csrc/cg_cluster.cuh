// One conjugate-gradient step's vector work in one kernel (internal to libsgpp_gb300): the two dot
// products and the three updates of a column run on one cluster of thread blocks, which exchange
// their partial sums through distributed shared memory. As separate kernels each dot product ends
// in a grid-wide reduction and the next kernel's launch; the vectors are short (a grid point per
// entry, 0.1 MB), so those launches and the serial sums of block partials took longer than the
// loads (17 us a step for one column of 2,561, 130 us for 16 of 4,159; now 5 and 7 us).
// Every sum has a fixed order: lanes by a butterfly, warps by a butterfly, blocks by rank.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sgmev {

constexpr int kCgCtas = 8;  // the portable cluster size
constexpr int kCgThreads = 512;

struct CgShared {
  double warp[kCgThreads / 32];
  double part[3];  // this block's sums, one slot per call so that no slot is written twice
};

// the cluster's sum of v, the same in every thread; `slot` 0, 1 or 2, each used once per kernel
__device__ __forceinline__ double cg_cluster_sum(double v, CgShared& sh, int slot) {
  namespace cg = cooperative_groups;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sh.warp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double w = lane < kCgThreads / 32 ? sh.warp[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane == 0) sh.part[slot] = w;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  double s = 0.0;
#pragma unroll
  for (int b = 0; b < kCgCtas; ++b) s += *cluster.map_shared_rank(&sh.part[slot], b);
  return s;
}

// no block leaves while another one may still read its shared memory
__device__ __forceinline__ void cg_cluster_end() { cooperative_groups::this_cluster().sync(); }

// thread's first entry and the stride over a column
__device__ __forceinline__ int64_t cg_first() {
  return static_cast<int64_t>(blockIdx.x % kCgCtas) * kCgThreads + threadIdx.x;
}
constexpr int64_t kCgStride = static_cast<int64_t>(kCgCtas) * kCgThreads;

// dq = d.q; alpha = dq != 0 ? delta / dq : 0; x += alpha d; r -= alpha q; rr = r.r; d = r + (rr / delta) d
__device__ __forceinline__ void cg_column_step(int64_t n, double* __restrict__ d,
                                               const double* __restrict__ q,
                                               double* __restrict__ x, double* __restrict__ r,
                                               double delta, CgShared& sh, double* dq_out,
                                               double* alpha_out, double* rr_out) {
  double acc = 0.0;
  for (int64_t i = cg_first(); i < n; i += kCgStride) acc = fma(d[i], q[i], acc);
  const double dq = cg_cluster_sum(acc, sh, 0);
  const double alpha = dq != 0.0 ? delta / dq : 0.0;
  acc = 0.0;
  for (int64_t i = cg_first(); i < n; i += kCgStride) {
    double ri = r[i];
    if (dq != 0.0) {
      x[i] = fma(alpha, d[i], x[i]);
      ri = fma(-alpha, q[i], ri);
      r[i] = ri;
    }
    acc = fma(ri, ri, acc);
  }
  const double rr = cg_cluster_sum(acc, sh, 1);
  const double beta = rr / delta;
  for (int64_t i = cg_first(); i < n; i += kCgStride) d[i] = fma(beta, d[i], r[i]);
  *dq_out = dq;
  *alpha_out = alpha;
  *rr_out = rr;
}

}  // namespace sgmev
