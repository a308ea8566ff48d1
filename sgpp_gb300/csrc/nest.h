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

struct NestPlan {
  bool ok = false;
  bool mod = false;
  int dim = 0, n_sub = 0, n_ent = 0, n_r = 0;
  int64_t n = 0, total = 0;
  std::vector<NestClass> classes;
  unsigned char* block = nullptr;  // device memory of the plan
  // device copies of NestTables
  int *lmax = nullptr, *facs = nullptr, *cuts = nullptr, *inv = nullptr, *clev = nullptr,
      *ccell = nullptr, *tinv = nullptr;
  NestOp4 *rops = nullptr, *qops = nullptr, *chunks = nullptr;
  NestOp2 *lops = nullptr, *cq = nullptr, *cs = nullptr;
  double* rows = nullptr;  // multTranspose: partial rows, per class [streams][row_len]
  int* bad = nullptr;      // flags of values that are not finite, one per block
  double* coef = nullptr;  // [total] coefficients in position order
  // tables of the data, built on the first product
  double* tab64 = nullptr;    // [n_ent][mpad]
  uint32_t* xcell = nullptr;  // [dim][mpad]
  cudaStream_t stream = nullptr;
};

// False (and a reason) when nest_plan does not take the grid or memory is short.
bool nest_build(NestPlan* p, int dim, int64_t n, const double* level_pow2, const double* index,
                bool mod, int num_sms, cudaStream_t stream, std::string* err);
void nest_free(NestPlan* p);

// The dense form of the operands, for coefficients or vectors that are not finite: such a value
// times a hat of 0 is NaN at every point outside the function's support, as in the dense kernels.
struct NestDense {
  const double* xt;
  const double2* li;
  int64_t mpad;
};

// out[j] = sum_g alpha_g phi_g(x_j), j in [j_begin, j_end) and the rest of their 64-point tiles,
// 0 beyond m; `part` holds part_elems partial sums
cudaError_t nest_mult64(NestPlan& p, cudaStream_t s, const NestDense& dense, int64_t m,
                        const double* alpha, double* out, int64_t j_begin, int64_t j_end,
                        double* part, int64_t part_elems, int num_sms, int* launches);

// out[g] (g < n; zero in [n, npad)) = sum_j v_j phi_g(x_j) (+ scale * add[g])
cudaError_t nest_multt64(NestPlan& p, cudaStream_t s, const NestDense& dense, int64_t m,
                         const double* v, int64_t npad, double* out, const double* add,
                         double scale, int num_sms, int* launches);

}  // namespace sgmev
