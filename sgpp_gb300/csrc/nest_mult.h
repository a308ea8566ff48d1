// The nested mult's kernels by dimension (internal interface of libsgpp_gb300; nest_mult.cu).
#pragma once

#include "nest.h"

namespace sgmev {

struct NestMultArgs {
  const NestOp4 *windows, *prog;
  int n_windows, words;  // windows of the list, words of the longest program
  int n_ent, dim;
  int entry[32], lmax[32];  // first table entry (level 2) and finest level of each dimension
  const float *tab_hi, *tab_lo;
  const double* tab64;
  const uint32_t* xcell;
  int64_t m, j_begin, n_tiles;
  float* out32;
  double* out64;
  void* part;
  int64_t out_end;  // outputs are written for j < out_end, zero beyond m
  NestDense dense;
  const int* inv;
  const double* alpha;
  int64_t n;
  const void* coef;  // coefficients in position order, or nullptr: gathered while they are staged
  int warps;         // warps of a CTA that take tiles; the others only help to stage
  const double* stop;  // device flag: when it is not 0 the product is skipped
};

// The launch of the mult in one precision, with its configuration in `c` on the first one; MD = dim up to
// kNestMacroDim, 0 for more dimensions. `spread`: see NestDense (always in FP64).
using NestMultLaunch = cudaError_t(NestPlan& p, cudaStream_t s, int precision, bool spread, NestConfig& c,
                                   NestMultArgs& a, int64_t mpad, int64_t part_bytes, int64_t tiles, int num_sms);
NestMultLaunch nest_mult_0, nest_mult_1, nest_mult_2, nest_mult_3, nest_mult_4, nest_mult_5, nest_mult_6,
    nest_mult_7, nest_mult_8, nest_mult_9, nest_mult_10, nest_mult_11, nest_mult_12, nest_mult_13,
    nest_mult_14, nest_mult_15, nest_mult_16;

}  // namespace sgmev
