// The nested mult (nest.cu has the method and the measurements): kernel, configuration and launch for
// NEST_MULT_DIM dimensions (0: more than kNestMacroDim). A translation unit per dimension, because the
// driver loads a unit's kernels together when the first of them is launched: with all dimensions in one
// unit the first mult of a process took 22 ms (d=8 level 4, 20,000 points), with its own alone 0.8.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "../../include/sgmev.h"
#include "nest_arith.cuh"
#include "nest_mult.h"
#include "subspace.h"

#ifndef NEST_MULT_DIM
#define NEST_MULT_DIM 0
#endif

namespace sgmev {
namespace {

// s += t * a with the rounding errors of s collected in c (FP32): the sums over groups and inner nodes, and
// over the dimensions where one forest or tree is all of the grid (regular ones of level 3 and 4), are long,
// and without this the error was up to 1.46 times that of the stored products, which are rounded once; now
// 0.7 to 1.06 times over 28 regular and four refined grids (d=12 level 4: 1.42 -> 1.02, adaptive d=8 level 4
// 1.43 -> 0.8). It costs 1 to 2 % (d=10 level 5, 262,147 points: 92.8 -> 94.3 us; 100 us with it in every forest and
// tree of such a grid, where the ratio is 0.9 without) and 3 to 5 % where a block is all of the grid (d=8 level 4,
// 262,144 points: 26.0 -> 26.9 us, 118 on stored products; d=16 level 3, whose kernel spills: 25.3 -> 29.1, 113).
template <typename V, int R>
__device__ __forceinline__ void mac_kept(V (&s)[R], V (&)[R], const V (&t)[R], const V (&a)[R]) { mac_all(s, t, a); }
__device__ __forceinline__ void mac_kept(float (&s)[2], float (&c)[2], const float (&t)[2], const float (&a)[2]) {
  // n = t a + s; c += t a + (s - n), where s - n is exact unless n is far smaller than s
  asm("{\n\t.reg .b64 vs, vt, va, vn, vd, vc, vm;\n\tmov.b64 vs, {%0, %1};\n\tmov.b64 vc, {%2, %3};\n\t"
      "mov.b64 vt, {%4, %5};\n\tmov.b64 va, {%6, %7};\n\tmov.b64 vm, {%8, %8};\n\t"
      "fma.rn.f32x2 vn, vt, va, vs;\n\tfma.rn.f32x2 vd, vn, vm, vs;\n\tfma.rn.f32x2 vd, vt, va, vd;\n\t"
      "add.rn.f32x2 vc, vc, vd;\n\tmov.b64 {%0, %1}, vn;\n\tmov.b64 {%2, %3}, vc;\n\t}"
      : "+f"(s[0]), "+f"(s[1]), "+f"(c[0]), "+f"(c[1])
      : "f"(t[0]), "f"(t[1]), "f"(a[0]), "f"(a[1]), "f"(-1.0f));
}
__device__ __forceinline__ void add(float& s, float v) { s += v; }
__device__ __forceinline__ void add(ff& s, ff v) { add_ff(s, v); }
// (a correction that is not finite belongs to a sum that is not)
__device__ __forceinline__ float corrected(float s, float c) { return fabsf(c) <= 3.4e38f ? s + c : s; }
__device__ __forceinline__ double corrected(double s, double) { return s; }
__device__ __forceinline__ ff corrected(ff s, ff) { return s; }
// asynchronous copies into shared memory: `bytes` (4 or 8) of a thread's own column
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
template <typename V>
__device__ __forceinline__ void prefetch_entry(const float* hi, const float* lo, const double* d, int64_t k) {
  if constexpr (std::is_same<V, double>::value) {
    prefetch_l2(d + k);
  } else {
    prefetch_l2(hi + k);
    if constexpr (sizeof(V) == 8) prefetch_l2(lo + k);
  }
}
// table entries of R adjacent points (k: the first one's index)
__device__ __forceinline__ void load_entry(float (&r)[2], const float* hi, const float*, const double*, int64_t k) { copy_async<8>(r, hi + k); }
__device__ __forceinline__ void load_entry(double (&r)[1], const float*, const float*, const double* d, int64_t k) { copy_async<8>(r, d + k); }
__device__ __forceinline__ void load_entry(ff (&r)[1], const float* hi, const float* lo, const double*, int64_t k) {
  copy_async<4>(&r[0].h, hi + k);
  copy_async<4>(&r[0].l, lo + k);
}

// coefficients into position order (launches that stage them more than once)
template <typename V>
__global__ void nest_coef_kernel(const double* __restrict__ alpha, const int* __restrict__ inv,
                                 int64_t total, V* __restrict__ coef) {
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < total;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int g = inv[p];
    set_val(coef[p], g >= 0 ? alpha[g] : 0.0);
  }
}

// NaN when a non-finite coefficient meets a hat of 0 at point j, else 0
template <typename V>
__device__ __noinline__ double mult_poison(const NestDense& d, int dim, int64_t n,
                                           const double* alpha, int64_t j) {
  double r = 0.0;
  for (int64_t g = 0; g < n; ++g) {
    const double a = held<V>(alpha[g]);
    if (!isfinite(a) && isnan(a * dense_value(d, dim, g, j))) r = a - a;
  }
  return r;
}
__device__ __forceinline__ void add_poison(float& s, double v) { s += static_cast<float>(v); }
__device__ __forceinline__ void add_poison(double& s, double v) { s += v; }
__device__ __forceinline__ void add_poison(ff& s, double v) { s.h += static_cast<float>(v); }

// R adjacent data points per thread (two in FP32, one in the wider arithmetics), a warp at a time over
// a contiguous range of 32 R-point tiles; the points' table rows and cells in shared memory
// ([entry][thread][R], private to the thread, copied asynchronously), their level-2 and level-3
// factors and cells in registers for the runs and trees (MD = dim, or 0 for more dimensions than
// kNestMacroDim: then the plan has none). A window's coefficients and program are staged in shared
// memory: a warp's 32 gathers from one row hit different banks or the same word, and the program's
// loads are broadcasts (read through L1 they missed half the time beside this much shared memory,
// and the FP32 kernel took 203 us instead of 128). blockIdx.y takes windows
// [y windows / splits, (y + 1) windows / splits) of the list and, with several splits, writes its own
// row of partial sums.
constexpr int kMultMaxThreads = 448;

// SPREAD: coefficients that are not finite spread as in the dense kernels. A variant of its own: as a
// branch of one kernel it cost the grids that need no look 1 to 2 %. WHOLE (FP32): one forest or tree is all of
// the grid, whose sums then carry their errors too (a variant for the same reason: 7 % as a branch).
template <typename V, int MD, bool SPREAD, bool WHOLE>
__global__ void __launch_bounds__(sizeof(V) == 4 ? 384 : kMultMaxThreads, 1)
    nest_mult_kernel(const __grid_constant__ NestMultArgs a) {
  if (a.stop && *a.stop != 0.0) return;
  constexpr int D = MD > 0 ? MD : 1, kV = sizeof(V), R = kPts<V>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, all = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = a.warps;
  const int nth = 32 * nw;
  const int64_t mpad = a.dense.mpad;
  using Col = V[R];
  using ColX = uint32_t[R];
  NestOp4* s_prog = reinterpret_cast<NestOp4*>(smem);
  Col* s_tab = reinterpret_cast<Col*>(s_prog + a.words) + tid;
  ColX* s_x = reinterpret_cast<ColX*>(s_tab - tid + a.n_ent * nth) + tid;
  V* s_coef = reinterpret_cast<V*>(s_x - tid + a.dim * nth);
  const int w_begin = blockIdx.y * a.n_windows / gridDim.y;
  const int w_end = (blockIdx.y + 1) * a.n_windows / gridDim.y;
  bool poison = false;  // a coefficient that is not finite (the same in every thread)
  auto stage = [&](const NestOp4& w) {
    for (int k = w.x + tid; k < w.y; k += all) s_prog[k - w.x] = a.prog[k];
    bool finite = true;
    if (a.coef) {
#pragma unroll 4
      for (int k = w.z + tid; k < w.w; k += all) {
        const V v = static_cast<const V*>(a.coef)[k];
        if constexpr (SPREAD) finite = finite && is_finite(v);
        s_coef[k - w.z] = v;
      }
    } else {
#pragma unroll 4
      for (int k = w.z + tid; k < w.w; k += all) {
        const int g = a.inv[k];
        V v;
        set_val(v, g >= 0 ? a.alpha[g] : 0.0);
        if constexpr (SPREAD) finite = finite && is_finite(v);
        s_coef[k - w.z] = v;
      }
    }
    if constexpr (SPREAD) poison = __syncthreads_or(!finite) || poison;
    else __syncthreads();
  };
  // the warps' tile ranges are contiguous and as equal as can be; every warp of the CTA runs the same
  // number of rounds (the barriers of several windows), some of them on no tile
  const int64_t warps = static_cast<int64_t>(gridDim.x) * nw, gw = static_cast<int64_t>(blockIdx.x) * nw + warp;
  const int64_t t_begin = warp < nw ? gw * a.n_tiles / warps : 0;
  const int64_t t_end = warp < nw ? (gw + 1) * a.n_tiles / warps : 0;
  const int64_t rounds = (a.n_tiles + warps - 1) / warps;
  const bool one = w_end - w_begin == 1;
  if (one) stage(a.windows[w_begin]);
  for (int64_t round = 0; round < rounds; ++round) {
    const bool live = t_begin + round < t_end;
    if (one && !live) break;
    const int64_t j = a.j_begin + ((t_begin + round) * 32 + lane) * R;
    V T2[D][R], T3[D][R];
    uint32_t B2[D][R], B3[D][R];  // byte offsets of the points' cells of levels 2 and 3
    if (live) {
#pragma unroll 4
      for (int t = 0; t < a.dim; ++t) copy_async<4 * R>(s_x[t * nth], a.xcell + t * mpad + j);
#pragma unroll 4
      for (int e = 0; e < a.n_ent; ++e)
        load_entry(s_tab[e * nth], a.tab_hi, a.tab_lo, a.tab64, e * mpad + j);
      // the warp's next tile into L2: it streams from HBM otherwise, a full latency per tile
      if (t_begin + round + 1 < t_end && (lane & 15) == 0) {
        const int64_t jn = j + 32 * R;
        for (int e = 0; e < a.n_ent; ++e) prefetch_entry<V>(a.tab_hi, a.tab_lo, a.tab64, e * mpad + jn);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      if constexpr (MD > 0) {
#pragma unroll
        for (int t = 0; t < MD; ++t) {
          const int bits = a.lmax[t] - 1;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const uint32_t x = s_x[t * nth][r];
            T2[t][r] = bits >= 1 ? s_tab[a.entry[t] * nth][r] : V{};
            B2[t][r] = bits >= 1 ? (x >> (bits - 1)) * kV : 0u;
            T3[t][r] = bits >= 2 ? s_tab[(a.entry[t] + 1) * nth][r] : V{};
            B3[t][r] = bits >= 2 ? (x >> (bits - 2)) * kV : 0u;
          }
        }
      }
    }
    V acc[R] = {}, acc_c[R] = {};
    for (int w = w_begin; w < w_end; ++w) {
      const NestOp4 win = a.windows[w];
      if (!one) {
        __syncthreads();  // the previous window is no longer read
        stage(win);
      }
      if (!live) continue;
      const NestOp4* op = s_prog;
      const NestOp4* const op_end = op + (win.y - win.x);
      while (op < op_end) {
        const NestOp4 head = *op++;
        V pr[R], ar[R] = {}, ar_c[R] = {};
        uint32_t cr[R] = {};
#pragma unroll
        for (int r = 0; r < R; ++r) set_val(pr[r], 1.0);
        const int* facs = reinterpret_cast<const int*>(op);
        for (int i = 0; i < head.y; ++i) {
          const int f = facs[i];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            pr[r] = mul(pr[r], s_tab[fac_e(f) * nth][r]);
            cr[r] = (cr[r] << fac_k(f)) | (s_x[fac_t(f) * nth][r] >> fac_shift(f));
          }
        }
        op += (head.y + 3) / 4;
        for (int q = 0; q < head.x; ++q) {
          const NestOp4 qo = op[0], qf = op[1];
          op += 2;
          uint32_t c[R];
          V tq[R], sum[R] = {};
#pragma unroll
          for (int r = 0; r < R; ++r) {
            tq[r] = s_tab[qf.x * nth][r];
            c[r] = (cr[r] << qf.z) | (s_x[qf.y * nth][r] >> qf.w);
          }
          if (MD == 0 || qo.y >= 0) {
            if (qo.x >= 0) {
#pragma unroll
              for (int r = 0; r < R; ++r) sum[r] = s_coef[qo.x + c[r]];
            }
            const NestOp4* const leaf_end = op + qo.y;
#pragma unroll 2
            for (; op < leaf_end; ++op) {
              const NestOp4 lo = *op;
              const int e = lo.y & 0xFFFF, t = lo.y >> 16;
#pragma unroll
              for (int r = 0; r < R; ++r)
                mac(sum[r], s_tab[e * nth][r],
                    s_coef[lo.x + ((c[r] << lo.z) | (s_x[t * nth][r] >> lo.w))]);
            }
          } else if constexpr (MD > 0) {
            const int kind = -qo.y - 1, t0 = kind >> 2;
            V sum_c[R] = {};
            auto ld = [](const char* p) { return *reinterpret_cast<const V*>(p); };
            // the value of a run and of a tree whose dimensions begin at t1, from their rows
            auto run = [&](const char* (&row)[R], int t1, V (&sr)[R]) {
#pragma unroll
              for (int r = 0; r < R; ++r) sr[r] = ld(row[r]);
#pragma unroll
              for (int t = MD - 1; t >= 0; --t) {
                if (t < t1) break;
                V v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = ld(row[r] + B2[t][r] + kV * (1 + 2 * (MD - 1 - t)));
                mac_all(sr, T2[t], v);
              }
            };
            // (`alone`, a constant where this is inlined: not one of a forest's, which adds them up. A
            // float-float tree then adds its level-2 and level-3 children apart: ModLinear, d=16 level 3,
            // 1.38 -> 1.11 times the error of the stored products, at 0.4 % of d=9 level 6's time)
            auto tree = [&](const char* (&row)[R], int t1, V (&st)[R], bool alone) {
              V s2[R] = {};
#pragma unroll
              for (int r = 0; r < R; ++r) st[r] = ld(row[r]);
#pragma unroll
              for (int t = MD - 1; t >= 0; --t) {
                if (t < t1) break;
                const int kt = MD - 1 - t, sec = kV * nest_tree_at(kt);
                V sq[R], v[R];
                const char* rq[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  rq[r] = row[r] + B2[t][r] * static_cast<uint32_t>(nest_run_row(kt));
                  sq[r] = ld(rq[r] + sec);
                  v[r] = ld(row[r] + B3[t][r] + (sec + kV * 2 * nest_run_row(kt)));
                }
                mac_all(st, T3[t], v);
#pragma unroll
                for (int u = MD - 1; u > t; --u) {
#pragma unroll
                  for (int r = 0; r < R; ++r) v[r] = ld(rq[r] + B2[u][r] + (sec + kV * (1 + 2 * (MD - 1 - u))));
                  mac_all(sq, T2[u], v);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) settle(sq[r]);
                if (WHOLE && alone) mac_kept(s2, sum_c, T2[t], sq);
                else if (std::is_same<V, ff>::value && alone) mac_all(s2, T2[t], sq);
                else mac_all(st, T2[t], sq);
              }
              if constexpr (WHOLE || std::is_same<V, ff>::value) {
                if (alone) {
#pragma unroll
                  for (int r = 0; r < R; ++r) add(st[r], s2[r]);
                }
              }
            };
            const char* row[R];
            if ((kind & 3) < 2) {
#pragma unroll
              for (int r = 0; r < R; ++r) row[r] = reinterpret_cast<const char*>(s_coef + qo.x + c[r] * qo.z);
              if ((kind & 3) == 0) run(row, t0, sum);
              else tree(row, t0, sum, true);
            } else {
              const V* cells = s_coef + qo.x;
#pragma unroll
              for (int r = 0; r < R; ++r) sum[r] = cells[c[r]];
              cells += ((1 << qo.z) + 3) & ~3;
              int tree_row = nest_tree_row(0), run_row = nest_run_row(0), tree_end = nest_tree_at(0);
              for (int t = MD - 1; t >= t0; --t) {
                const int bits = a.lmax[t] - 1;
                const Col* te = s_tab + a.entry[t] * nth;
                V v[R], tl[R];
                uint32_t x[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  x[r] = s_x[t * nth][r];
                  row[r] = reinterpret_cast<const char*>(cells + ((c[r] << 1) | (x[r] >> (bits - 1))) * tree_row);
                  tl[r] = te[0][r];
                }
                tree(row, t + 1, v, false);
#pragma unroll
                for (int r = 0; r < R; ++r) settle(v[r]);
                if (WHOLE) mac_kept(sum, sum_c, tl, v);
                else mac_all(sum, tl, v);
                cells += (2 * tree_row) << qo.z;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  row[r] = reinterpret_cast<const char*>(cells + ((c[r] << 2) | (x[r] >> (bits - 2))) * run_row);
                  tl[r] = te[nth][r];
                }
                run(row, t + 1, v);
#pragma unroll
                for (int r = 0; r < R; ++r) settle(v[r]);
                if (WHOLE) mac_kept(sum, sum_c, tl, v);
                else mac_all(sum, tl, v);
                cells += (4 * run_row) << qo.z;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  v[r] = cells[(c[r] << 3) | (x[r] >> (bits - 3))];
                  tl[r] = te[2 * nth][r];
                }
                if (WHOLE) mac_kept(sum, sum_c, tl, v);
                else mac_all(sum, tl, v);
                cells += 8 << qo.z;
                // the next dimension's row lengths (nest_tree_at, nest_tree_row and nest_run_row of k + 1)
                tree_end += 2 * run_row + 4;
                tree_row = ((tree_end + 3) & ~7) + 4;
                const int k = MD - t;
                run_row = 2 * k + ((k & 1) == 0 ? 2 : 4);
              }
            }
            if constexpr (WHOLE) mac_all(ar_c, tq, sum_c);
          }
#pragma unroll
          for (int r = 0; r < R; ++r) settle(sum[r]);
          mac_kept(ar, ar_c, tq, sum);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) settle(ar[r]);
        mac_kept(acc, acc_c, pr, ar);
        if constexpr (std::is_same<V, float>::value) mac_all(acc_c, pr, ar_c);
      }
    }
    if (!live) continue;
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = corrected(acc[r], acc_c[r]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t k = j + r;
      const bool real = k < a.m;
      if (SPREAD && poison && real) add_poison(acc[r], mult_poison<V>(a.dense, a.dim, a.n, a.alpha, k));
      if (gridDim.y > 1) {
        reinterpret_cast<V*>(a.part)[blockIdx.y * mpad + k] = acc[r];
      } else {
        if (a.out32 && k < a.out_end) a.out32[k] = real ? static_cast<float>(to_double(acc[r])) : 0.0f;
        if (a.out64 && k < a.out_end) a.out64[k] = real ? to_double(acc[r]) : 0.0;
      }
    }
  }
}

// Threads per CTA, the window list and the CTAs that share a tile of points, once per operator (m
// does not change). A CTA has as many warps as its shared memory holds table rows for (one CTA per
// SM), or fewer when the tiles would not reach every SM. Of the lists, the one with the least cycles
// by a model of the measured kernels: a round of a warp costs about 2,500 cycles for its table rows
// and 75 (FP32, two points a thread), 150 (float-float) or 21 a warp of the SM (FP64, whose pipe the
// warps share) per subspace; staging a window about 1,500 and a cycle per 40 bytes; several CTAs per
// tile pay about 5,000 for the partial sums' pass.
template <typename V, typename Kern>
cudaError_t mult_config(const NestPlan& p, NestConfig* c, Kern kern, int64_t m, int64_t mpad,
                        int64_t part_bytes, int num_sms) {
  constexpr int64_t kV = sizeof(V), R = kPts<V>;
  const int caps = kV == 4 ? 0 : kNestLists / 2;
  const int64_t tiles = std::max<int64_t>(1, (m + 32 * R - 1) / (32 * R));
  const int64_t row = 32 * R * (kV * p.n_ent + 4 * p.dim);  // table rows of a warp
  const int64_t most = (kV == 4 ? 384 : kMultMaxThreads) / 32;
  double best = 0.0;
  int64_t warps = 1, window = 0;
  for (int k = 0; k < kNestLists / 2; ++k) {
    const int list = caps + k, n_windows = p.lists[list + 1] - p.lists[list];
    const int64_t ctas = nest_list_ctas(list);
    if (k > 0 && (n_windows < ctas || part_bytes < ctas * mpad * kV)) break;
    const int64_t w = kV * p.list_cells[list] + static_cast<int64_t>(sizeof(NestOp4)) * p.list_words[list];
    const int64_t fit = std::max<int64_t>(1, std::min<int64_t>({most, (static_cast<int64_t>(kNestMultSmem) - w) / row,
                                                                std::max<int64_t>(2, (tiles * ctas + num_sms - 1) / num_sms)}));
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((tiles + fit - 1) / fit, num_sms / ctas));
    const int64_t rounds = (tiles + blocks * fit - 1) / (blocks * fit);
    const double per_sub = std::is_same<V, double>::value ? 21.0 * static_cast<double>(fit) : kV == 4 ? 75.0 : 150.0;
    const double staged = 1500.0 + static_cast<double>(kV * p.list_cells[list]) / 40.0;
    const int64_t per_cta = (n_windows + ctas - 1) / ctas;
    const double cost = static_cast<double>(rounds) * (2500.0 + 20.0 * p.n_ent + per_sub * p.n_sub / static_cast<double>(ctas)) +
                        static_cast<double>(per_cta > 1 ? rounds * per_cta : 1) * staged + (ctas > 1 ? 5000.0 : 0.0);
    if (k == 0 || cost < best) {
      best = cost;
      c->list = list;
      c->splits = static_cast<int>(ctas);
      c->restage = per_cta > 1 && rounds > 1;
      warps = fit;
      window = w;
    }
  }
  c->warps = static_cast<int>(warps);
  c->threads = 32 * std::max(8, c->warps);
  c->smem = static_cast<size_t>(window + row * warps);
  cudaError_t e = set_smem_cap(kern, c->smem);
  int per_sm = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, c->threads, c->smem);
  if (e != cudaSuccess) return e;
  c->ctas = std::max(1, per_sm) * num_sms;
  return cudaSuccess;
}

template <typename V, int MD, bool SPREAD, bool WHOLE = false>
cudaError_t launch_mult(NestPlan& p, cudaStream_t s, NestConfig& c, NestMultArgs& a, int64_t mpad,
                        int64_t part_bytes, int64_t tiles, int num_sms) {
  auto kern = nest_mult_kernel<V, MD, SPREAD, WHOLE>;
  if (c.threads == 0) {
    const cudaError_t e = mult_config<V>(p, &c, kern, a.m, mpad, part_bytes, num_sms);
    if (e != cudaSuccess) {
      c.threads = 0;
      return e;
    }
  }
  a.windows = p.windows + p.lists[c.list];
  a.n_windows = p.lists[c.list + 1] - p.lists[c.list];
  a.words = p.list_words[c.list];
  a.warps = c.warps;
  a.coef = nullptr;
  if (c.restage) {
    nest_coef_kernel<V><<<32, 512, 0, s>>>(a.alpha, p.inv, p.total, static_cast<V*>(p.coef));
    a.coef = p.coef;
  }
  const int nw = c.warps;
  const int64_t blocks = std::max<int64_t>(
      1, std::min<int64_t>((tiles + nw - 1) / nw, c.ctas / c.splits));
  kern<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(c.splits)), c.threads, c.smem, s>>>(a);
  return cudaGetLastError();
}
}  // namespace

#define NEST_MULT_NAME_(d) nest_mult_##d
#define NEST_MULT_NAME(d) NEST_MULT_NAME_(d)
cudaError_t NEST_MULT_NAME(NEST_MULT_DIM)(NestPlan& p, cudaStream_t s, int precision, bool spread, NestConfig& c,
                                          NestMultArgs& a, int64_t mpad, int64_t part_bytes, int64_t tiles,
                                          int num_sms) {
  constexpr int D = NEST_MULT_DIM;
  if (precision == SGMEV_FP64) return launch_mult<double, D, true>(p, s, c, a, mpad, part_bytes, tiles, num_sms);
  if (precision == SGMEV_FP32) {
    // (grids whose values spread are mostly small: one variant, with everything)
    constexpr bool kBlocks = D > 0;
    if (spread) return launch_mult<float, D, true, kBlocks>(p, s, c, a, mpad, part_bytes, tiles, num_sms);
    if (p.whole && !p.plain) return launch_mult<float, D, false, kBlocks>(p, s, c, a, mpad, part_bytes, tiles, num_sms);
    return launch_mult<float, D, false>(p, s, c, a, mpad, part_bytes, tiles, num_sms);
  }
  return spread ? launch_mult<ff, D, true>(p, s, c, a, mpad, part_bytes, tiles, num_sms)
                : launch_mult<ff, D, false>(p, s, c, a, mpad, part_bytes, tiles, num_sms);
}

}  // namespace sgmev
