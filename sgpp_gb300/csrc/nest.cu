// Nested subspace products.
//
// The dense kernels evaluate every grid point's basis function for every data point (in FP64 3 d
// instructions per pair, at 1/62 of FP32's rate); the materialised ones stream a product per subspace
// and point from HBM. Exactly one function per subspace can be non-zero at a point (the reference's
// DEFAULT operator evaluates only those, base/src/sgpp/base/algorithm/AlgorithmEvaluation.hpp:129-179),
// and the functions of subspaces that share active dimensions share factors. So the subspaces form a
// tree (nest_plan.h), a point's one-dimensional factors are tabulated once per data set, and
//   mult   nests the sum: result = H_1 sum over the tree, each node costing one multiply-add,
//              sum_r P_r sum_{q below r} T_q (a_q + sum_{leaf c below q} T_c a_c)
//          with groups r (their product P_r is formed once), inner nodes q (children of r that have
//          children) and the leaves below q; whole subtrees of up to three more levels, which is most
//          of a regular grid, run as unrolled code on registers;
//   multT  forms v_j P_q for the inner nodes of a tile of points in shared memory and then, one
//          thread per subspace, adds (v_j P_q) T into the thread's own cells: one multiply-add per
//          subspace and point, in a fixed order.
// Bound: FP64 the FP64 pipe (2 lanes per clock and SM), at about 1.3 instructions per subspace and
// point; FP32 and float-float instruction issue (7 instructions per subspace and point in FP32, 28 in
// float-float, at 0.55 of the issue rate with the 12 to 14 warps per SM that the tables leave room
// for). Measured before and after:
//   FP64, d=5 level 6 (252 subspaces), 65,536 points: mult 10,791 -> 36 us, multT 10,895 -> 57 us
//   FP64, adaptive d=8 grid (4,024 points), 2^19 data points: B^T (B a) 199.1 -> 1.22 ms
//   FP32, d=10 level 5 (1,001 subspaces), 262,147 points: mult 168 -> 94 us (materialised before)
//   float-float, d=9 level 6 (2,002 subspaces), 40,961 points: mult 583 -> 109 us (hats on the fly)
// The errors against 64-bit results, relative to their norm: FP64 mult 6.1e-16 before and after,
// multT 6.2e-16 -> 4.4e-16; FP32 mult 1.1e-7 -> 1.1e-7 (0.7 to 1.06 times the stored products' over 32
// grids); float-float 1.5e-13 -> 8e-15 (0.05 to 0.3 times the stored
// products' over 14 grids, ModLinear 0.4 to 1.1).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <utility>

#include "../../include/sgmev.h"
#include "devmem.h"
#include "kernels.cuh"
#include "nest_arith.cuh"
#include "nest_mult.h"
#include "subspace.h"

namespace sgmev {
namespace {

constexpr int kTile = kNestTile;
// ---- tables -----------------------------------------------------------------------------------
// One thread per data point. The hats of a dimension follow one another by the tent map,
// h_{l+1} = 2 min(h_l, 1 - h_l), which is exact in floating point (the smaller side is h_l itself or
// an exact difference by Sterbenz's lemma), from h_1 = 2 min(x, 1 - x). A point outside (0, 1)^d
// (or closer to a face than 2^-1000) has H_1 = 0 and the table of the cube's centre.
template <bool MOD, bool F64, bool F32>
__global__ void nest_table_kernel(const double* __restrict__ xt, int64_t mpad, int64_t m, int dim,
                                  const int* __restrict__ lmax, double* __restrict__ tab64,
                                  float* __restrict__ tab_hi, float* __restrict__ tab_lo,
                                  uint32_t* __restrict__ xcell) {
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= mpad) return;
  auto put = [&](int e, double v) {
    if constexpr (F64) tab64[e * mpad + j] = v;
    if constexpr (F32) {
      const float hi = static_cast<float>(v);
      tab_hi[e * mpad + j] = hi;
      tab_lo[e * mpad + j] = static_cast<float>(v - static_cast<double>(hi));
    }
  };
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
        put(e, h);
      }
    } else {
      double h = 2.0 * (x > 0.5 ? 1.0 - x : x);
      h1p *= h;
      const double r = 1.0 / h;
      for (int l = 2; l <= bits + 1; ++l, ++e) {
        h = 2.0 * (h > 0.5 ? 1.0 - h : h);
        put(e, h * r);
      }
    }
  }
  put(0, h1p);
}

// ---- multTranspose -----------------------------------------------------------------------------
// CTA (stream, chunk): chunk's subspaces over the stream's contiguous range of tiles. Phase A: lane
// = point, a warp per inner node, one depth of the tree after the other. Phase B: thread =
// subspace, points in order, sums in the thread's own cells. LONG: FP32 streams of more than 1,024
// points, which a plain FP32 sum would round by up to 2^-12 (8,192 points in one: 1.2e-4 off at worst); a
// variant of its own, as the branch in the other one made that 2 to 4 us slower (d=10 level 5, 34 us).
struct NestMulttArgs {
  const NestOp4* chunks;
  const NestOp2 *cq, *cs, *cwarp;
  const int *clev, *ccell;
  const float *tab_hi, *tab_lo;
  const double* tab64;
  const uint32_t* xcell;
  int64_t mpad, m, n_tiles, row_len;
  int n_ent, dim, nq_max, sums, streams;
  double* rows;
  int* bad;
  const double* stop;
  bool spread;  // values that are not finite spread as in the dense kernels
};
__device__ __forceinline__ void read_entry(float& r, const NestMulttArgs& a, int64_t k) { r = a.tab_hi[k]; }
__device__ __forceinline__ void read_entry(double& r, const NestMulttArgs& a, int64_t k) { r = a.tab64[k]; }
__device__ __forceinline__ void read_entry(ff& r, const NestMulttArgs& a, int64_t k) { r = ff{a.tab_hi[k], a.tab_lo[k]}; }

template <typename V, typename VIN, bool LONG>
__global__ void __launch_bounds__(256) nest_multt_kernel(const __grid_constant__ NestMulttArgs a,
                                                         const VIN* __restrict__ v) {
  if (a.stop && *a.stop != 0.0) return;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nth >> 5;
  const int chunk = blockIdx.x / a.streams, stream = blockIdx.x - chunk * a.streams;
  const NestTileLayout lay(a.nq_max, a.n_ent, a.dim);
  V* s_acc = reinterpret_cast<V*>(smem);
  V* s_p = s_acc + a.sums;
  V* s_t = s_p + kTile * lay.qs;
  uint32_t* s_x = reinterpret_cast<uint32_t*>(s_t + kTile * lay.es);
  uint16_t* s_c = reinterpret_cast<uint16_t*>(s_x + kTile * lay.xs);
  const NestOp4 ch = a.chunks[chunk];
  const NestOp2 own = a.cs[chunk * nth + tid];
  const int own_cells = a.ccell[chunk * nth + tid];
  const int own_e = fac_e(own.y), own_t = fac_t(own.y), own_k = fac_k(own.y),
            own_s = fac_shift(own.y);
  const NestOp2 at = a.cwarp[chunk * nw + warp];
  V* const own_acc = s_acc + at.x + lane;  // cell c at 32 c
  for (int c = 0; c < own_cells; ++c) own_acc[32 * c] = V{};
  bool nonfinite = false;
  const int64_t t_begin = stream * a.n_tiles / a.streams, t_end = (stream + 1) * a.n_tiles / a.streams;
  for (int64_t tile = t_begin; tile < t_end; ++tile) {
    const int64_t j0 = tile * kTile;
    __syncthreads();  // phase B of the previous tile is done
    for (int e = warp; e < a.n_ent; e += nw) read_entry(s_t[lane * lay.es + e], a, e * a.mpad + j0 + lane);
    for (int t = warp; t < a.dim; t += nw) s_x[lane * lay.xs + t] = a.xcell[t * a.mpad + j0 + lane];
    if (warp == nw - 1) {  // the root: v_j H_1 (the same warp reads H_1 itself)
      const double vj = j0 + lane < a.m ? static_cast<double>(v[j0 + lane]) : 0.0;
      V h1, vv;
      read_entry(h1, a, j0 + lane);
      set_val(vv, vj);
      nonfinite = nonfinite || !is_finite(vv);
      V root = mul(vv, h1);
      if constexpr (std::is_same<V, float>::value) {
        // (rounded once instead of three times: the sums' error, against that of the stored products, 1.22 -> 1.09
        // times with d=8 level 6 and 8,000 points, 0.7 -> 0.6 with d=4..16 level 3)
        if (is_finite(vv))
          root = static_cast<float>(vj * (static_cast<double>(h1) + static_cast<double>(a.tab_lo[j0 + lane])));
      }
      s_p[lane * lay.qs] = root;
      s_c[lane * lay.cs] = 0;
      set_val(s_t[lane * lay.es + a.n_ent], 1.0);
    }
    __syncthreads();
    for (int d = 0; d < ch.w; ++d) {
      const int q_end = a.clev[ch.z + d + 1];
      for (int q = a.clev[ch.z + d] + warp; q < q_end; q += nw) {
        const NestOp2 o = a.cq[ch.x + q];
        s_p[lane * lay.qs + q] = mul(s_p[lane * lay.qs + o.x], s_t[lane * lay.es + fac_e(o.y)]);
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
        V* acc = own_acc + 32 * c;
        V r = *acc;
        mac(r, s_p[i * lay.qs + own.x], s_t[i * lay.es + own_e]);
        *acc = r;
      }
      // every 1,024 points float-float sums are settled, and FP32 ones of LONG streams go into the FP64 row
      if (std::is_same<V, ff>::value && ((tile - t_begin) & 31) == 31)
        for (int c = 0; c < own_cells; ++c) settle(own_acc[32 * c]);
      if constexpr (LONG) {
        if (((tile - t_begin) & 31) == 31 && tile + 1 < t_end) {
          double* row = a.rows + stream * a.row_len + at.y + lane;
          for (int c = 0; c < own_cells; ++c) {
            const double s = to_double(own_acc[32 * c]);
            row[32 * c] = tile >= t_begin + 32 ? row[32 * c] + s : s;
            own_acc[32 * c] = V{};
          }
        }
      }
    }
  }
  double* row = a.rows + stream * a.row_len + at.y + lane;
  for (int c = 0; c < own_cells; ++c) {
    const double s = to_double(own_acc[32 * c]);
    if constexpr (LONG) row[32 * c] = t_end - t_begin > 32 ? row[32 * c] + s : s;
    else row[32 * c] = s;
  }
  const int any = __syncthreads_or(a.spread && nonfinite);
  if (tid == 0) a.bad[blockIdx.x] = any;
}

// NaN when a non-finite v_j meets a hat of 0 of grid point g, else 0
template <typename V, typename VIN>
__device__ __noinline__ double multt_poison(const NestDense& d, int dim, int64_t m,
                                            const VIN* v, int64_t g) {
  double r = 0.0;
  for (int64_t j = 0; j < m; ++j) {
    const double vj = held<V>(static_cast<double>(v[j]));
    if (!isfinite(vj) && isnan(vj * dense_value(d, dim, g, j))) r = vj - vj;
  }
  return r;
}

// out[g] = sum over the streams' rows in a fixed order (+ scale add[g]): a block of 32 x 8 threads
// takes 32 positions; thread (x, y) adds rows y, y + 8, ... in order, then the 8 sums in y order
constexpr int kSumGroups = 8;
template <typename V, typename VIN>
__global__ void __launch_bounds__(32 * kSumGroups) nest_finish_kernel(
    const double* __restrict__ rows, int nrows, int64_t row_len, const int* __restrict__ tinv,
    const double* __restrict__ add, double scale, double* __restrict__ out,
    const int* __restrict__ bad, NestDense dense, int dim, int64_t m,
    const VIN* __restrict__ v) {
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
    if (poison) r += multt_poison<V>(dense, dim, m, v, g);
    out[g] = add ? fma(scale, add[g], r) : r;
  }
}

}  // namespace

bool nest_build(NestPlan* p, int dim, int64_t n, const double* level_pow2, const double* index,
                bool mod, int num_sms, cudaStream_t stream, std::string* err, size_t* need) {
  nest_free(p);
  *need = 0;
  p->stream = stream;
  NestTables h;
  if (!nest_plan(&h, dim, n, level_pow2, index, err)) return false;
  p->dim = dim;
  p->n = n;
  p->mod = mod;
  p->n_sub = h.n_sub;
  p->n_act = h.n_act;
  p->cells = h.cells;
  p->cmax = h.cmax;
  p->whole = h.whole;
  p->n_ent = h.n_ent;
  p->lists = h.list_begin;
  p->list_cells = h.list_cells;
  p->list_words = h.list_words;
  for (int t = 0, e = 1; t < dim; ++t) {
    p->h_entry[t] = e;
    p->h_lmax[t] = h.lmax[t];
    e += h.lmax[t] - 1;
  }
  p->total = static_cast<int64_t>(h.inv.size());
  p->classes = h.classes;
  int flags = 4 * num_sms;
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
  put(&p->windows, h.windows);
  put(&p->prog, h.prog);
  put(&p->inv, h.inv);
  put(&p->chunks, h.chunks);
  put(&p->cq, h.cq);
  put(&p->clev, h.clev);
  put(&p->cs, h.cs);
  put(&p->cwarp, h.cwarp);
  put(&p->ccell, h.ccell);
  put(&p->tinv, h.tinv);
  const size_t o_coef = (host.size() + 255) / 256 * 256,
               o_bad = o_coef + sizeof(double) * h.inv.size();
  if (dev_malloc(&p->block, o_bad + sizeof(int) * flags, stream) != cudaSuccess ||
      cudaMemcpyAsync(p->block, host.data(), host.size(), cudaMemcpyHostToDevice, stream) !=
          cudaSuccess) {  // (pageable source: the copy has taken the data when it returns)
    (void)cudaGetLastError();
    nest_free(p);
    *need = o_bad + sizeof(int) * flags;
    *err = "nested plan allocation failed";
    return false;
  }
  for (const auto& k : at) *k.first = p->block + k.second;
  p->coef = p->block + o_coef;
  p->bad = reinterpret_cast<int*>(p->block + o_bad);
  p->ok = true;
  return true;
}

void nest_free(NestPlan* p) {
  void* ptrs[] = {p->block, p->rows[0], p->rows[1], p->rows[2], p->tab64, p->tab_hi, p->xcell};
  for (void* q : ptrs) dev_free(q, p->stream);
  *p = NestPlan{};
}

bool nest_built(const NestPlan& p, int precision, bool transpose) {
  return p.ok && (precision == SGMEV_FP64 ? p.tab64 != nullptr : p.tab_hi != nullptr) &&
         (!transpose || !p.streams[precision].empty());
}

namespace {
// the tables that the precision reads, built on its first product
cudaError_t tables(NestPlan& p, cudaStream_t s, const NestDense& d, int64_t m, bool f64,
                   int* launches) {
  if (f64 ? p.tab64 != nullptr : p.tab_hi != nullptr) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  const int64_t n = p.n_ent * d.mpad, cells = sizeof(uint32_t) * p.dim * d.mpad;
  const bool first = !p.xcell;
  if (first) e = dev_malloc(&p.xcell, cells, s);
  if (e == cudaSuccess) e = f64 ? dev_malloc(&p.tab64, sizeof(double) * n, s) : dev_malloc(&p.tab_hi, 2 * sizeof(float) * n, s);
  if (e != cudaSuccess) {
    p.need = sizeof(double) * n + (first ? cells : 0);
    if (first) dev_free(p.xcell, s);
    if (first) p.xcell = nullptr;
    return e;
  }
  const unsigned blocks = static_cast<unsigned>((d.mpad + 127) / 128);
  auto kern = f64 ? (p.mod ? nest_table_kernel<true, true, false> : nest_table_kernel<false, true, false>)
                  : (p.mod ? nest_table_kernel<true, false, true> : nest_table_kernel<false, false, true>);
  kern<<<blocks, 128, 0, s>>>(d.xt, d.mpad, m, p.dim, p.lmax, p.tab64, p.tab_hi,
                              p.tab_hi ? p.tab_hi + n : nullptr, p.xcell);
  ++*launches;
  return cudaGetLastError();
}

template <typename V, typename TP>
cudaError_t mult(NestPlan& p, cudaStream_t s, NestConfig& c, const NestDense& dense, int64_t m,
                 const double* alpha, float* out32, double* out64, int64_t j_begin, int64_t j_end,
                 int64_t out_end, void* part, int64_t part_bytes, int num_sms, bool spread,
                 int* launches) {
  constexpr bool kF64 = std::is_same<V, double>::value;
  cudaError_t e = tables(p, s, dense, m, kF64, launches);
  if (e != cudaSuccess) return e;
  constexpr int64_t kTilePts = 32 * kPts<V>;
  j_begin = j_begin / kTilePts * kTilePts;  // mpad is a multiple of 1024
  j_end = (j_end + kTilePts - 1) / kTilePts * kTilePts;
  NestMultArgs a;
  a.prog = p.prog;
  a.n_ent = p.n_ent;
  a.dim = p.dim;
  for (int t = 0; t < 32; ++t) {
    a.entry[t] = t < p.dim ? p.h_entry[t] : 0;
    a.lmax[t] = t < p.dim ? p.h_lmax[t] : 1;
  }
  a.tab_hi = p.tab_hi;
  a.tab_lo = p.tab_hi ? p.tab_hi + p.n_ent * dense.mpad : nullptr;
  a.tab64 = p.tab64;
  a.xcell = p.xcell;
  a.m = m;
  a.j_begin = j_begin;
  a.n_tiles = (j_end - j_begin) / kTilePts;
  a.out32 = out32;
  a.out64 = out64;
  a.part = part;
  a.out_end = out_end;
  a.stop = p.stop;
  a.dense = dense;
  a.inv = p.inv;
  a.alpha = alpha;
  a.n = p.n;
  static NestMultLaunch* const launch[kNestMacroDim + 1] = {
      nest_mult_0,  nest_mult_1,  nest_mult_2,  nest_mult_3,  nest_mult_4,  nest_mult_5,
      nest_mult_6,  nest_mult_7,  nest_mult_8,  nest_mult_9,  nest_mult_10, nest_mult_11,
      nest_mult_12, nest_mult_13, nest_mult_14, nest_mult_15, nest_mult_16};
  const int precision = kF64 ? SGMEV_FP64 : std::is_same<V, float>::value ? SGMEV_FP32 : SGMEV_DF64;
  e = launch[p.dim <= kNestMacroDim ? p.dim : 0](p, s, precision, spread, c, a, dense.mpad, part_bytes,
                                                  a.n_tiles, num_sms);
  if (e != cudaSuccess) return e;
  *launches += c.restage ? 2 : 1;
  if (c.splits > 1) {
    const unsigned blocks = static_cast<unsigned>((j_end - j_begin + 255) / 256);
    if (out64)
      reduce_splits_kernel<TP, double><<<blocks, 256, 0, s>>>(static_cast<const TP*>(part), c.splits, dense.mpad, j_begin,
                                                              std::min(m, j_end), std::min(out_end, j_end), out64, nullptr, 0.0);
    if (out32)
      reduce_splits_kernel<TP, float><<<blocks, 256, 0, s>>>(static_cast<const TP*>(part), c.splits, dense.mpad, j_begin,
                                                             std::min(m, j_end), std::min(out_end, j_end), out32, nullptr, 0.0);
    ++*launches;
  }
  return cudaGetLastError();
}
}  // namespace

cudaError_t nest_mult(NestPlan& p, cudaStream_t s, int precision, const NestDense& dense, int64_t m,
                      const double* alpha, float* out32, double* out64, int64_t j_begin,
                      int64_t j_end, int64_t out_end, void* part, int64_t part_bytes, int num_sms,
                      bool spread, int* launches) {
  NestConfig& c = p.config[precision == SGMEV_FP32 && p.plain ? 3 : precision];  // (a kernel each)
  switch (precision) {
    case SGMEV_FP64:
      return mult<double, double>(p, s, c, dense, m, alpha, out32, out64, j_begin, j_end, out_end, part, part_bytes, num_sms, spread, launches);
    case SGMEV_FP32:
      return mult<float, float>(p, s, c, dense, m, alpha, out32, out64, j_begin, j_end, out_end, part, part_bytes, num_sms, spread, launches);
    default:
      return mult<ff, float2>(p, s, c, dense, m, alpha, out32, out64, j_begin, j_end, out_end, part, part_bytes, num_sms, spread, launches);
  }
}

namespace {
// the multTranspose's streams and partial rows in the precision
template <typename V>
cudaError_t multt_rows(NestPlan& p, cudaStream_t s, int precision, int64_t m, int num_sms) {
  if (!p.streams[precision].empty()) return cudaSuccess;
  auto kern = nest_multt_kernel<V, double, false>;
  const int64_t n_tiles = std::max<int64_t>(1, (m + kTile - 1) / kTile);
  // as many streams as fit the SMs at once (at most 256 MB of rows); fixed from here on, and
  // with them the order of every sum
  std::vector<int> st;
  int64_t elems = 0;
  for (const NestClass& c : p.classes) {
    const size_t sm = c.smem(sizeof(V), p.n_ent, p.dim);
    cudaError_t e = set_smem_cap(kern, sm);
    if constexpr (std::is_same<V, float>::value) {
      if (e == cudaSuccess) e = set_smem_cap(nest_multt_kernel<float, float, false>, sm);
      if (e == cudaSuccess) e = set_smem_cap(nest_multt_kernel<float, double, true>, sm);
      if (e == cudaSuccess) e = set_smem_cap(nest_multt_kernel<float, float, true>, sm);
    }
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, c.threads, sm);
    if (e != cudaSuccess) return e;
    const int64_t resident = std::min<int64_t>(4, std::max(1, per_sm)) * num_sms;
    st.push_back(static_cast<int>(std::max<int64_t>(
        1, std::min<int64_t>({resident / c.chunks, n_tiles, (int64_t(1) << 25) / c.row_len}))));
    elems += st.back() * c.row_len;
  }
  const cudaError_t e = dev_malloc(&p.rows[precision], sizeof(double) * elems, s);
  if (e == cudaSuccess) p.streams[precision] = st;
  else p.need = sizeof(double) * elems;
  return e;
}

template <typename V, typename VIN>
cudaError_t multt(NestPlan& p, cudaStream_t s, int precision, const NestDense& dense, int64_t m, const VIN* v,
                  int64_t npad, double* out, const double* add, double scale, bool spread, int* launches) {
  const std::vector<int>& streams = p.streams[precision];
  double* rows = p.rows[precision];
  cudaError_t e = cudaSuccess;
  const int64_t n_tiles = std::max<int64_t>(1, (m + kTile - 1) / kTile);
  if (npad > p.n) {
    e = cudaMemsetAsync(out + p.n, 0, sizeof(double) * (npad - p.n), s);
    if (e != cudaSuccess) return e;
  }
  NestMulttArgs a;
  a.cq = p.cq;
  a.clev = p.clev;
  a.tab_hi = p.tab_hi;
  a.tab_lo = p.tab_hi ? p.tab_hi + p.n_ent * dense.mpad : nullptr;
  a.tab64 = p.tab64;
  a.xcell = p.xcell;
  a.mpad = dense.mpad;
  a.m = m;
  a.n_tiles = n_tiles;
  a.n_ent = p.n_ent;
  a.dim = p.dim;
  a.bad = p.bad;
  a.stop = p.stop;
  a.spread = spread;
  a.rows = rows;
  int64_t cs_at = 0;
  for (size_t k = 0; k < p.classes.size(); ++k) {
    const NestClass& c = p.classes[k];
    a.chunks = p.chunks + c.chunk_begin;
    a.cs = p.cs + cs_at;
    a.ccell = p.ccell + cs_at;
    a.nq_max = c.nq;
    a.cwarp = p.cwarp + cs_at / 32;
    a.sums = c.sums;
    a.streams = streams[k];
    a.row_len = c.row_len;
    auto kern = nest_multt_kernel<V, VIN, false>;
    if constexpr (std::is_same<V, float>::value)
      if ((n_tiles + streams[k] - 1) / streams[k] > 32) kern = nest_multt_kernel<V, VIN, true>;
    kern<<<static_cast<unsigned>(streams[k] * c.chunks), c.threads, c.smem(sizeof(V), p.n_ent, p.dim), s>>>(a, v);
    nest_finish_kernel<V, VIN><<<static_cast<unsigned>((c.row_len + 31) / 32), dim3(32, kSumGroups), 0, s>>>(
        a.rows, streams[k], c.row_len, p.tinv + c.row_begin, add, scale, out, p.bad, dense, p.dim, m, v);
    a.rows += streams[k] * c.row_len;
    cs_at += static_cast<int64_t>(c.chunks) * c.threads;
    *launches += 2;
  }
  return cudaGetLastError();
}
}  // namespace

bool nest_prepare(NestPlan& p, cudaStream_t s, int precision, bool transpose, const NestDense& dense,
                  int64_t m, int num_sms, int* launches) {
  bool& refused = p.refused[transpose ? 1 : 0][precision];
  if (refused) return false;
  cudaError_t e = tables(p, s, dense, m, precision == SGMEV_FP64, launches);
  if (e == cudaSuccess && transpose)
    e = precision == SGMEV_FP64   ? multt_rows<double>(p, s, precision, m, num_sms)
        : precision == SGMEV_DF64 ? multt_rows<ff>(p, s, precision, m, num_sms)
                                  : multt_rows<float>(p, s, precision, m, num_sms);
  if (e != cudaSuccess) (void)cudaGetLastError();
  refused = e != cudaSuccess;
  return !refused;
}

cudaError_t nest_multt(NestPlan& p, cudaStream_t s, int precision, const NestDense& dense, int64_t m,
                       const double* v64, const float* v32, int64_t npad, double* out,
                       const double* add, double scale, bool spread, int* launches) {
  if (precision == SGMEV_FP64)
    return multt<double>(p, s, precision, dense, m, v64, npad, out, add, scale, spread, launches);
  if (precision == SGMEV_DF64)
    return multt<ff>(p, s, precision, dense, m, v64, npad, out, add, scale, spread, launches);
  if (v32) return multt<float>(p, s, precision, dense, m, v32, npad, out, add, scale, spread, launches);
  return multt<float>(p, s, precision, dense, m, v64, npad, out, add, scale, spread, launches);
}

}  // namespace sgmev
