// Nested subspace products in FP64.
//
// The dense kernels evaluate every grid point's basis function for every data point: 3 d FP64
// instructions per pair, and GB300's FP64 rate is 1/62 of FP32's. Exactly one function per
// subspace can be non-zero at a point (the reference's DEFAULT operator evaluates only those,
// base/src/sgpp/base/algorithm/AlgorithmEvaluation.hpp:129-179), and the functions of subspaces
// that share active dimensions share factors. So the subspaces form a tree (nest.h), a point's
// one-dimensional factors are tabulated once per data set, and
//   mult   nests the sum: result = H_1 sum over the tree, each node costing one multiply-add,
//              sum_r P_r sum_{q below r} T_q (a_q + sum_{leaf c below q} T_c a_c)
//          with groups r (their product P_r is formed once), inner nodes q (children of r that have
//          children) and the leaves below q;
//   multT  forms v_j P_q for the inner nodes of a tile of points in shared memory and then, one
//          thread per subspace, adds (v_j P_q) T into the thread's own cells: one multiply-add per
//          subspace and point, in a fixed order.
// Bound: the FP64 pipe (2 lanes per clock and SM), at about 1.3 instructions per subspace and
// point against 3 d per grid point and point of the dense kernels. d=5 level 6 (5,503 points, 252
// subspaces), 65,536 data points: mult 10,791 -> 43 us, multTranspose 10,895 -> 60 us; B^T(B a) on an
// adaptive d=8 grid (4,024 points), 2^19 data points: 199.1 -> 1.46 ms. The error against 64-bit
// sums is that of the dense kernels (mult 6.0e-16 against 5.9e-16, multTranspose 4.0e-16 against
// 5.6e-16 of the result's norm).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <utility>

#include "devmem.h"
#include "kernels.cuh"
#include "nest.h"
#include "subspace.h"

namespace sgmev {
namespace {

constexpr int kMultThreads = kNestMultThreads, kTile = kNestTile;
constexpr int kBadBlocks = 32;  // blocks of the coefficient gather

// ---- tables -----------------------------------------------------------------------------------
// One thread per data point. The hats of a dimension follow one another by the tent map,
// h_{l+1} = 2 min(h_l, 1 - h_l), which is exact in floating point (the smaller side is h_l itself or
// an exact difference by Sterbenz's lemma), from h_1 = 2 min(x, 1 - x). A point outside (0, 1)^d
// (or closer to a face than 2^-1000) has H_1 = 0 and the table of the cube's centre.
template <bool MOD>
__global__ void nest_table_kernel(const double* __restrict__ xt, int64_t mpad, int64_t m, int dim,
                                  const int* __restrict__ lmax, double* __restrict__ tab,
                                  uint32_t* __restrict__ xcell) {
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= mpad) return;
  bool inside = j < m;
  for (int t = 0; t < dim; ++t) {
    const double x = xt[t * mpad + j];
    inside = inside && (MOD ? x >= 0.0 && x <= 1.0 : x > 0x1p-1000 && x < 1.0);
  }
  double h1p = inside ? 1.0 : 0.0;
  int e = 1;
  for (int t = 0; t < dim; ++t) {
    const double x = inside ? xt[t * mpad + j] : 0.5;
    const int bits = lmax[t] - 1;
    const uint32_t last = (1u << bits) - 1u;
    const uint32_t c = min(static_cast<uint32_t>(x * static_cast<double>(1u << bits)), last);
    xcell[t * mpad + j] = c;
    if constexpr (MOD) {
      for (int l = 2; l <= bits + 1; ++l, ++e) {
        const double L = static_cast<double>(1u << l), y = x * L;
        const uint32_t k = c >> (bits - (l - 1)), top = (1u << (l - 1)) - 1u;
        double h;
        if (k == 0u) h = 2.0 - y;
        else if (k == top) h = y - (L - 2.0);
        else h = 1.0 - fabs(y - static_cast<double>(2u * k + 1u));
        tab[e * mpad + j] = h;
      }
    } else {
      double h = 2.0 * (x > 0.5 ? 1.0 - x : x);
      h1p *= h;
      const double r = 1.0 / h;
      for (int l = 2; l <= bits + 1; ++l, ++e) {
        h = 2.0 * (h > 0.5 ? 1.0 - h : h);
        tab[e * mpad + j] = h * r;
      }
    }
  }
  tab[j] = h1p;
}

// ---- mult ----------------------------------------------------------------------------------------
// coefficients into position order; bad[block] = a coefficient that is not finite was seen
__global__ void nest_coef_kernel(const double* __restrict__ alpha, const int* __restrict__ inv,
                                 int64_t total, double* __restrict__ coef, int* __restrict__ bad) {
  bool b = false;
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < total;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int g = inv[p];
    const double a = g >= 0 ? alpha[g] : 0.0;
    coef[p] = a;
    b = b || !isfinite(a);
  }
  const int any = __syncthreads_or(b);
  if (threadIdx.x == 0) bad[blockIdx.x] = any;
}

// the dense value of grid point g's function at point j (0 exactly outside its support)
template <bool MOD>
__device__ double dense_value(const NestDense& d, int dim, int64_t g, int64_t j) {
  double p = h_first<MOD>(d.xt[j], d.li[g * dim]);
  for (int t = 1; t < dim; ++t) p = h_next<MOD>(p, d.xt[t * d.mpad + j], d.li[g * dim + t]);
  return p;
}

// NaN when a non-finite coefficient meets a hat of 0 at point j, else 0
template <bool MOD>
__device__ __noinline__ double mult_poison(const NestDense& d, int dim, int64_t n,
                                           const double* alpha, int64_t j) {
  double r = 0.0;
  for (int64_t g = 0; g < n; ++g) {
    const double a = alpha[g];
    if (!isfinite(a) && isnan(a * dense_value<MOD>(d, dim, g, j))) r = a - a;
  }
  return r;
}

// One thread per data point; its table row and cells in shared memory ([entry][thread], private to
// the thread). The program is the same for all threads, so its loads are broadcasts; the
// coefficients are gathered through L1 (a subspace's cells are contiguous). blockIdx.y takes the
// groups [cuts[y], cuts[y + 1]) and writes its own row of `out`.
template <bool MOD>
__global__ void __launch_bounds__(kMultThreads) nest_mult64_kernel(
    const NestOp4* __restrict__ rops, const int* __restrict__ facs, const NestOp4* __restrict__ qops,
    const NestOp2* __restrict__ lops, const int* __restrict__ cuts, const double* __restrict__ coef,
    const double* __restrict__ tab, const uint32_t* __restrict__ xcell, int n_ent, int dim,
    int64_t m, int64_t j_begin, int64_t out_stride, double* __restrict__ out,
    const int* __restrict__ bad, NestDense dense, const double* __restrict__ alpha, int64_t n) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x;
  const int64_t mpad = dense.mpad;
  const int64_t j = j_begin + static_cast<int64_t>(blockIdx.x) * kMultThreads + tid;
  double* s_tab = reinterpret_cast<double*>(smem) + tid;
  uint32_t* s_x = reinterpret_cast<uint32_t*>(smem + sizeof(double) * n_ent * kMultThreads) + tid;
#pragma unroll 8
  for (int e = 0; e < n_ent; ++e) s_tab[e * kMultThreads] = tab[e * mpad + j];
#pragma unroll 4
  for (int t = 0; t < dim; ++t) s_x[t * kMultThreads] = xcell[t * mpad + j];
  double acc = 0.0;
  const int r_end = cuts[blockIdx.y + 1];
  for (int r = cuts[blockIdx.y]; r < r_end; ++r) {
    const NestOp4 ro = rops[r];
    double pr = 1.0;
    uint32_t cr = 0;
    for (int i = ro.z; i < ro.w; ++i) {
      const int f = facs[i];
      pr *= s_tab[fac_e(f) * kMultThreads];
      cr = (cr << fac_k(f)) | (s_x[fac_t(f) * kMultThreads] >> fac_shift(f));
    }
    double ar = 0.0;
    for (int q = ro.x; q < ro.y; ++q) {
      const NestOp4 qo = qops[q];
      const uint32_t c = (cr << fac_k(qo.w)) | (s_x[fac_t(qo.w) * kMultThreads] >> fac_shift(qo.w));
      double sum = qo.x >= 0 ? __ldg(coef + qo.x + c) : 0.0;
#pragma unroll 4
      for (int i = qo.y; i < qo.z; ++i) {
        const NestOp2 lo = lops[i];
        const uint32_t cl =
            (c << fac_k(lo.y)) | (s_x[fac_t(lo.y) * kMultThreads] >> fac_shift(lo.y));
        sum = fma(s_tab[fac_e(lo.y) * kMultThreads], __ldg(coef + lo.x + cl), sum);
      }
      ar = fma(s_tab[fac_e(qo.w) * kMultThreads], sum, ar);
    }
    acc = fma(pr, ar, acc);
  }
  if (blockIdx.y == 0 && __syncthreads_or(tid < kBadBlocks && bad[tid] != 0) && j < m)
    acc += mult_poison<MOD>(dense, dim, n, alpha, j);
  out[blockIdx.y * out_stride + j] = j < m ? acc : 0.0;
}

// ---- multTranspose -----------------------------------------------------------------------------
// CTA (stream, chunk): chunk's subspaces over the stream's contiguous range of tiles. Phase A: lane
// = point, a warp per inner node, one depth of the tree after the other. Phase B: thread =
// subspace, points in order, sums in the thread's own cells.
__global__ void __launch_bounds__(256) nest_multt64_kernel(
    const NestOp4* __restrict__ chunks, const NestOp2* __restrict__ cq, const int* __restrict__ clev,
    const NestOp2* __restrict__ cs, const int* __restrict__ ccell, const double* __restrict__ tab,
    const uint32_t* __restrict__ xcell, int64_t mpad, int64_t m, int n_ent, int dim, int nq_max,
    int cells, const double* __restrict__ v, int64_t n_tiles, int streams, int64_t row_len,
    double* __restrict__ rows, int* __restrict__ bad) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nth >> 5;
  const int chunk = blockIdx.x / streams, stream = blockIdx.x - chunk * streams;
  const NestTileLayout lay(nq_max, n_ent, dim);
  double* s_acc = reinterpret_cast<double*>(smem);
  double* s_p = s_acc + static_cast<size_t>(cells) * nth;
  double* s_t = s_p + kTile * lay.qs;
  uint32_t* s_x = reinterpret_cast<uint32_t*>(s_t + kTile * lay.es);
  uint16_t* s_c = reinterpret_cast<uint16_t*>(s_x + kTile * lay.xs);
  const NestOp4 ch = chunks[chunk];
  const NestOp2 own = cs[chunk * nth + tid];
  const int own_cells = ccell[chunk * nth + tid];
  const int own_e = fac_e(own.y), own_t = fac_t(own.y), own_k = fac_k(own.y),
            own_s = fac_shift(own.y);
  for (int c = 0; c < own_cells; ++c) s_acc[c * nth + tid] = 0.0;
  bool nonfinite = false;
  const int64_t t_end = (stream + 1) * n_tiles / streams;
  for (int64_t tile = stream * n_tiles / streams; tile < t_end; ++tile) {
    const int64_t j0 = tile * kTile;
    __syncthreads();  // phase B of the previous tile is done
    for (int e = warp; e < n_ent; e += nw) s_t[lane * lay.es + e] = tab[e * mpad + j0 + lane];
    for (int t = warp; t < dim; t += nw) s_x[lane * lay.xs + t] = xcell[t * mpad + j0 + lane];
    if (warp == nw - 1) {  // the root: v_j H_1 (the same warp reads H_1 itself)
      const double vj = j0 + lane < m ? v[j0 + lane] : 0.0;
      nonfinite = nonfinite || !isfinite(vj);
      s_p[lane * lay.qs] = vj * tab[j0 + lane];
      s_c[lane * lay.cs] = 0;
      s_t[lane * lay.es + n_ent] = 1.0;
    }
    __syncthreads();
    for (int d = 0; d < ch.w; ++d) {
      const int q_end = clev[ch.z + d + 1];
      for (int q = clev[ch.z + d] + warp; q < q_end; q += nw) {
        const NestOp2 o = cq[ch.x + q];
        s_p[lane * lay.qs + q] = s_p[lane * lay.qs + o.x] * s_t[lane * lay.es + fac_e(o.y)];
        s_c[lane * lay.cs + q] = static_cast<uint16_t>(
            (static_cast<uint32_t>(s_c[lane * lay.cs + o.x]) << fac_k(o.y)) |
            (s_x[lane * lay.xs + fac_t(o.y)] >> fac_shift(o.y)));
      }
      __syncthreads();
    }
    if (own_cells > 0) {
#pragma unroll 8
      for (int i = 0; i < kTile; ++i) {
        const uint32_t c = (static_cast<uint32_t>(s_c[i * lay.cs + own.x]) << own_k) |
                           (s_x[i * lay.xs + own_t] >> own_s);
        double* a = s_acc + c * nth + tid;
        *a = fma(s_p[i * lay.qs + own.x], s_t[i * lay.es + own_e], *a);
      }
    }
  }
  double* row = rows + stream * row_len + static_cast<int64_t>(chunk) * cells * nth;
  for (int c = 0; c < own_cells; ++c) row[c * nth + tid] = s_acc[c * nth + tid];
  const int any = __syncthreads_or(nonfinite);
  if (tid == 0) bad[blockIdx.x] = any;
}

// NaN when a non-finite v_j meets a hat of 0 of grid point g, else 0
template <bool MOD>
__device__ __noinline__ double multt_poison(const NestDense& d, int dim, int64_t m,
                                            const double* v, int64_t g) {
  double r = 0.0;
  for (int64_t j = 0; j < m; ++j)
    if (!isfinite(v[j]) && isnan(v[j] * dense_value<MOD>(d, dim, g, j))) r = v[j] - v[j];
  return r;
}

// out[g] = sum over the streams' rows in a fixed order (+ scale add[g]): a block of 32 x 8 threads
// takes 32 positions; thread (x, y) adds rows y, y + 8, ... in order, then the 8 sums in y order
constexpr int kSumGroups = 8;
template <bool MOD>
__global__ void __launch_bounds__(32 * kSumGroups) nest_finish_kernel(
    const double* __restrict__ rows, int nrows, int64_t row_len, const int* __restrict__ tinv,
    const double* __restrict__ add, double scale, double* __restrict__ out,
    const int* __restrict__ bad, NestDense dense, int dim, int64_t m,
    const double* __restrict__ v) {
  __shared__ double part[kSumGroups][33];
  const int64_t k = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
  const int y = threadIdx.y, tid = y * 32 + threadIdx.x;
  const int g = k < row_len ? tinv[k] : -1;
  double a = 0.0;
  if (g >= 0) {
#pragma unroll 4
    for (int b = y; b < nrows; b += kSumGroups) a += rows[b * row_len + k];
  }
  part[y][threadIdx.x] = a;
  bool flagged = false;
  for (int b = tid; b < nrows; b += 32 * kSumGroups) flagged = flagged || bad[b] != 0;
  const int poison = __syncthreads_or(flagged);
  if (y == 0 && g >= 0) {
    double r = part[0][threadIdx.x];
    for (int b = 1; b < kSumGroups; ++b) r += part[b][threadIdx.x];
    if (poison) r += multt_poison<MOD>(dense, dim, m, v, g);
    out[g] = add ? fma(scale, add[g], r) : r;
  }
}

}  // namespace

bool nest_build(NestPlan* p, int dim, int64_t n, const double* level_pow2, const double* index,
                bool mod, int num_sms, cudaStream_t stream, std::string* err) {
  nest_free(p);
  p->stream = stream;
  NestTables h;
  if (!nest_plan(&h, dim, n, level_pow2, index, err)) return false;
  p->dim = dim;
  p->n = n;
  p->mod = mod;
  p->n_sub = h.n_sub;
  p->n_ent = h.n_ent;
  p->n_r = static_cast<int>(h.rops.size());
  p->total = static_cast<int64_t>(h.inv.size());
  p->classes = h.classes;
  int flags = std::max(kBadBlocks, 4 * num_sms);
  for (const NestClass& c : h.classes) flags = std::max(flags, c.chunks);
  // one allocation and one copy for the whole plan: the operator may live for a single product
  std::vector<unsigned char> host;
  std::vector<std::pair<void**, size_t>> at;
  auto put = [&](auto** dst, const auto& src) {
    const size_t o = (host.size() + 255) / 256 * 256, bytes = sizeof(src[0]) * src.size();
    host.resize(o + bytes);
    std::memcpy(host.data() + o, src.data(), bytes);
    at.emplace_back(reinterpret_cast<void**>(dst), o);
  };
  put(&p->lmax, h.lmax);
  put(&p->rops, h.rops);
  put(&p->facs, h.facs);
  put(&p->qops, h.qops);
  put(&p->lops, h.lops);
  put(&p->cuts, h.cuts);
  put(&p->inv, h.inv);
  put(&p->chunks, h.chunks);
  put(&p->cq, h.cq);
  put(&p->clev, h.clev);
  put(&p->cs, h.cs);
  put(&p->ccell, h.ccell);
  put(&p->tinv, h.tinv);
  const size_t o_coef = (host.size() + 255) / 256 * 256,
               o_bad = o_coef + sizeof(double) * h.inv.size();
  if (dev_malloc(&p->block, o_bad + sizeof(int) * flags, stream) != cudaSuccess ||
      cudaMemcpyAsync(p->block, host.data(), host.size(), cudaMemcpyHostToDevice, stream) !=
          cudaSuccess) {  // (pageable source: the copy has taken the data when it returns)
    (void)cudaGetLastError();
    nest_free(p);
    *err = "nested plan allocation failed";
    return false;
  }
  for (const auto& k : at) *k.first = p->block + k.second;
  p->coef = reinterpret_cast<double*>(p->block + o_coef);
  p->bad = reinterpret_cast<int*>(p->block + o_bad);
  p->ok = true;
  return true;
}

void nest_free(NestPlan* p) {
  void* ptrs[] = {p->block, p->rows, p->tab64, p->xcell};
  for (void* q : ptrs) dev_free(q, p->stream);
  *p = NestPlan{};
}

namespace {
cudaError_t tables(NestPlan& p, cudaStream_t s, const NestDense& d, int64_t m, int* launches) {
  if (p.tab64) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  if (!p.xcell) e = dev_malloc(&p.xcell, sizeof(uint32_t) * p.dim * d.mpad, s);
  if (e == cudaSuccess) e = dev_malloc(&p.tab64, sizeof(double) * p.n_ent * d.mpad, s);
  if (e != cudaSuccess) return e;
  const unsigned blocks = static_cast<unsigned>((d.mpad + 127) / 128);
  auto kern = p.mod ? nest_table_kernel<true> : nest_table_kernel<false>;
  kern<<<blocks, 128, 0, s>>>(d.xt, d.mpad, m, p.dim, p.lmax, p.tab64, p.xcell);
  ++*launches;
  return cudaGetLastError();
}
}  // namespace

cudaError_t nest_mult64(NestPlan& p, cudaStream_t s, const NestDense& dense, int64_t m,
                        const double* alpha, double* out, int64_t j_begin, int64_t j_end,
                        double* part, int64_t part_elems, int num_sms, int* launches) {
  cudaError_t e = tables(p, s, dense, m, launches);
  if (e != cudaSuccess) return e;
  j_begin = j_begin / kMultThreads * kMultThreads;  // whole tiles; mpad is a multiple of them
  j_end = (j_end + kMultThreads - 1) / kMultThreads * kMultThreads;
  nest_coef_kernel<<<kBadBlocks, 512, 0, s>>>(alpha, p.inv, p.total, p.coef, p.bad);
  const size_t sm = (sizeof(double) * p.n_ent + sizeof(uint32_t) * p.dim) * kMultThreads;
  auto kern = p.mod ? nest_mult64_kernel<true> : nest_mult64_kernel<false>;
  e = set_smem_cap(kern, sm);
  if (e != cudaSuccess) return e;
  // few tiles of points: several CTAs share the groups of one tile, so that every SM has work. The
  // count comes from the whole data set, so that a range gives the bits of the full product.
  const int64_t tiles_all = (m + kMultThreads - 1) / kMultThreads;
  int64_t splits = std::min<int64_t>({kNestSplits, 4 * num_sms / std::max<int64_t>(tiles_all, 1),
                                      p.n_sub / 32, p.n_r, part_elems / dense.mpad});
  splits = std::max<int64_t>(1, splits);
  const dim3 grid(static_cast<unsigned>((j_end - j_begin) / kMultThreads),
                  static_cast<unsigned>(splits));
  kern<<<grid, kMultThreads, sm, s>>>(
      p.rops, p.facs, p.qops, p.lops, p.cuts + (splits - 1) * (kNestSplits + 1), p.coef, p.tab64,
      p.xcell, p.n_ent, p.dim, m, j_begin, dense.mpad, splits > 1 ? part : out, p.bad, dense, alpha,
      p.n);
  *launches += 2;
  if (splits > 1) {
    const unsigned blocks = static_cast<unsigned>((j_end - j_begin + 255) / 256);
    reduce_splits_kernel<double, double><<<blocks, 256, 0, s>>>(
        part, static_cast<int>(splits), dense.mpad, j_begin, std::min(m, j_end), j_end, out, nullptr, 0.0);
    ++*launches;
  }
  return cudaGetLastError();
}

cudaError_t nest_multt64(NestPlan& p, cudaStream_t s, const NestDense& dense, int64_t m,
                         const double* v, int64_t npad, double* out, const double* add,
                         double scale, int num_sms, int* launches) {
  cudaError_t e = tables(p, s, dense, m, launches);
  if (e != cudaSuccess) return e;
  const int64_t n_tiles = std::max<int64_t>(1, (m + kTile - 1) / kTile);
  if (!p.rows) {
    // as many streams as fit the SMs at once (at most 256 MB of rows); fixed from here on, and
    // with them the order of every sum
    int64_t elems = 0;
    for (NestClass& c : p.classes) {
      e = set_smem_cap(nest_multt64_kernel, c.smem);
      int per_sm = 0;
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nest_multt64_kernel, c.threads, c.smem);
      if (e != cudaSuccess) return e;
      const int64_t resident = std::min<int64_t>(4, std::max(1, per_sm)) * num_sms;
      c.streams = static_cast<int>(std::max<int64_t>(
          1, std::min<int64_t>({resident / c.chunks, n_tiles, (int64_t(1) << 25) / c.row_len})));
      elems += c.streams * c.row_len;
    }
    e = dev_malloc(&p.rows, sizeof(double) * elems, s);
    if (e != cudaSuccess) return e;
  }
  if (npad > p.n) {
    e = cudaMemsetAsync(out + p.n, 0, sizeof(double) * (npad - p.n), s);
    if (e != cudaSuccess) return e;
  }
  double* rows = p.rows;
  int64_t cs_at = 0;
  for (const NestClass& c : p.classes) {
    nest_multt64_kernel<<<static_cast<unsigned>(c.streams * c.chunks), c.threads, c.smem, s>>>(
        p.chunks + c.chunk_begin, p.cq, p.clev, p.cs + cs_at, p.ccell + cs_at, p.tab64, p.xcell,
        dense.mpad, m, p.n_ent, p.dim, c.nq, c.cells, v, n_tiles, c.streams, c.row_len, rows, p.bad);
    auto fin = p.mod ? nest_finish_kernel<true> : nest_finish_kernel<false>;
    fin<<<static_cast<unsigned>((c.row_len + 31) / 32), dim3(32, kSumGroups), 0, s>>>(
        rows, c.streams, c.row_len, p.tinv + c.row_begin, add, scale, out, p.bad, dense, p.dim, m, v);
    rows += c.streams * c.row_len;
    cs_at += static_cast<int64_t>(c.chunks) * c.threads;
    *launches += 2;
  }
  return cudaGetLastError();
}

}  // namespace sgmev
