// Nested subspace products (internal interface of libsgpp_gb300): one basis function per subspace
// and data point, with the one-dimensional factors of a point tabulated once and the products of
// the subspaces sharing their common factors.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "nest_plan.h"

namespace sgmev {

struct NestConfig {  // launch of the mult in one precision, fixed on its first product
  int threads = 0, warps = 0, list = 0, splits = 1, ctas = 0;
  bool restage = false;  // coefficients in position order first: they are staged several times
  size_t smem = 0;
};

struct NestPlan {
  const double* stop = nullptr;  // device flag: when it is not 0 the products are skipped
  bool plain = false;            // FP32 mult of an inner solve: sums as they come where one block is the grid
  bool ok = false;
  bool mod = false;
  int dim = 0, n_sub = 0, n_ent = 0;
  int64_t n = 0, total = 0;
  int64_t n_act = 0, cells = 0;  // see NestTables
  int cmax = 0;
  bool whole = false;
  std::vector<NestClass> classes;
  std::vector<int> lists, list_cells, list_words;  // see NestTables
  int h_entry[32] = {0}, h_lmax[32] = {0};
  NestConfig config[4];  // by precision (SGMEV_FP64, SGMEV_FP32, SGMEV_DF64); FP32 plain
  std::vector<int> streams[3];  // multTranspose: tile streams (rows of partial sums) of each class
  unsigned char* block = nullptr;  // device memory of the plan
  // device copies of NestTables
  int *lmax = nullptr, *inv = nullptr, *clev = nullptr, *ccell = nullptr, *tinv = nullptr;
  NestOp4 *windows = nullptr, *prog = nullptr, *chunks = nullptr;
  NestOp2 *cq = nullptr, *cs = nullptr, *cwarp = nullptr;
  double* rows[3] = {nullptr, nullptr, nullptr};  // multTranspose: partial rows, per class [streams][row_len]
  void* coef = nullptr;    // [total] coefficients in position order, in the product's precision
  int* bad = nullptr;      // flags of values that are not finite, one per block
  // tables of the data, built on the first product
  double* tab64 = nullptr;    // [n_ent][mpad], FP64 products
  float* tab_hi = nullptr;    // [2][n_ent][mpad], high and low parts, FP32 and float-float products
  uint32_t* xcell = nullptr;  // [dim][mpad]
  bool refused[2][3] = {};  // by direction and precision: nest_prepare() found no memory
  size_t need = 0;          // for so many bytes
  cudaStream_t stream = nullptr;
};

// False (and a reason) when nest_plan does not take the grid, or with *need bytes where device memory is short.
bool nest_build(NestPlan* p, int dim, int64_t n, const double* level_pow2, const double* index,
                bool mod, int num_sms, cudaStream_t stream, std::string* err, size_t* need);
void nest_free(NestPlan* p);
// whether the product needs nothing more to be built (a product under stream capture must not)
bool nest_built(const NestPlan& p, int precision, bool transpose);

// The dense form of the operands, for coefficients or vectors that are not finite: such a value
// times a hat of 0 is NaN at every point outside the function's support, as in the dense kernels
// (products with `spread` set; the others, like the subspace kernels, meet a value only in its cell).
struct NestDense {
  const double* xt;
  const double2* li;
  int64_t mpad;
  bool mod;  // ModLinear
};

// Builds what a product of the precision needs beside the plan: the tables of the data and, for the
// transpose, its partial rows. False when there is no memory for them, `need` bytes (not tried again
// while `refused` is set).
bool nest_prepare(NestPlan& p, cudaStream_t s, int precision, bool transpose, const NestDense& dense,
                  int64_t m, int num_sms, int* launches);

// out32[j] and / or out64[j] = sum_g alpha_g phi_g(x_j) in the given precision (SGMEV_FP64, SGMEV_FP32,
// SGMEV_DF64), j in [j_begin, j_end) and the rest of their tiles (32 points, 64 in FP32) up to
// out_end, 0 beyond m; alpha [n] FP64;
// `part` holds part_bytes of partial sums
cudaError_t nest_mult(NestPlan& p, cudaStream_t s, int precision, const NestDense& dense, int64_t m,
                      const double* alpha, float* out32, double* out64, int64_t j_begin,
                      int64_t j_end, int64_t out_end, void* part, int64_t part_bytes, int num_sms,
                      bool spread, int* launches);

// out[g] (g < n; zero in [n, npad)) = sum_j v_j phi_g(x_j) (+ scale * add[g]) in the given precision;
// v64 [m], or v32 [m] (nullptr: v64) for SGMEV_FP32
cudaError_t nest_multt(NestPlan& p, cudaStream_t s, int precision, const NestDense& dense, int64_t m,
                       const double* v64, const float* v32, int64_t npad, double* out,
                       const double* add, double scale, bool spread, int* launches);

}  // namespace sgmev
