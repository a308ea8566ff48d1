// The three arithmetics of the nested products (internal to libsgpp_gb300), and the dense form of a basis
// function for values that are not finite.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.cuh"
#include "nest.h"

namespace sgmev {
namespace {

// The three arithmetics. A value of the float-float one is (h, l) as in kernels.cuh.
__device__ __forceinline__ void set_val(float& r, double v) { r = static_cast<float>(v); }
__device__ __forceinline__ void set_val(double& r, double v) { r = v; }
__device__ __forceinline__ void set_val(ff& r, double v) {
  r.h = static_cast<float>(v);
  r.l = static_cast<float>(v - static_cast<double>(r.h));
}
// s += t * a
__device__ __forceinline__ void mac(float& s, float t, float a) { s = fmaf(t, a, s); }
__device__ __forceinline__ void mac(double& s, double t, double a) { s = fma(t, a, s); }
__device__ __forceinline__ void mac(ff& s, ff t, ff a) { add_ff(s, mul_ff(t, a)); }
template <typename V, int R>
__device__ __forceinline__ void mac_all(V (&s)[R], const V (&t)[R], const V (&a)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) mac(s[r], t[r], a[r]);
}
// two FP32 multiply-adds in one instruction
__device__ __forceinline__ void mac_all(float (&s)[2], const float (&t)[2], const float (&a)[2]) {
  asm("{\n\t.reg .b64 vs, vt, va;\n\tmov.b64 vs, {%0, %1};\n\tmov.b64 vt, {%2, %3};\n\tmov.b64 va, {%4, %5};\n\t"
      "fma.rn.f32x2 vs, vt, va, vs;\n\tmov.b64 {%0, %1}, vs;\n\t}"
      : "+f"(s[0]), "+f"(s[1]) : "f"(t[0]), "f"(t[1]), "f"(a[0]), "f"(a[1]));
}
__device__ __forceinline__ float mul(float a, float b) { return a * b; }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ ff mul(ff a, ff b) {
  ff r = mul_ff(a, b);
  renorm_ff(r);
  return r;
}
// a finished sum, before it becomes a factor (mul_ff drops the product of the low parts)
__device__ __forceinline__ void settle(float&) {}
__device__ __forceinline__ void settle(double&) {}
__device__ __forceinline__ void settle(ff& s) { renorm_ff(s); }
__device__ __forceinline__ double to_double(float v) { return static_cast<double>(v); }
__device__ __forceinline__ double to_double(double v) { return v; }
__device__ __forceinline__ double to_double(ff v) {
  return static_cast<double>(v.h) + static_cast<double>(v.l);
}
__device__ __forceinline__ bool is_finite(float v) { return isfinite(v); }
__device__ __forceinline__ bool is_finite(double v) { return isfinite(v); }
__device__ __forceinline__ bool is_finite(ff v) { return isfinite(v.h); }
// the dense value of grid point g's function at point j (0 exactly outside its support)
template <bool MOD>
__device__ double dense_value(const NestDense& d, int dim, int64_t g, int64_t j) {
  double p = h_first<MOD>(d.xt[j], d.li[g * dim]);
  for (int t = 1; t < dim; ++t) p = h_next<MOD>(p, d.xt[t * d.mpad + j], d.li[g * dim + t]);
  return p;
}
__device__ double dense_value(const NestDense& d, int dim, int64_t g, int64_t j) {
  return d.mod ? dense_value<true>(d, dim, g, j) : dense_value<false>(d, dim, g, j);
}

// a value as the product's arithmetic holds it
template <typename V>
__device__ __forceinline__ double held(double v) {
  V r;
  set_val(r, v);
  return to_double(r);
}

// adjacent data points per thread of the mult
template <typename V>
constexpr int kPts = sizeof(V) == 4 ? 2 : 1;

}  // namespace
}  // namespace sgmev
