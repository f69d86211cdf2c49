// What the float64 lensing integrals (jcg_tracer64.cu, jcg_gradfront64.cu) share:
// pairs of signed and scaled doubles, and comoving distances from the node.
#pragma once

#include "jcg_internal.cuh"
#include "jcg_px.cuh"

namespace jcg {

constexpr int T64_RUN = 8;                       // points per run
constexpr int T64_RUNS = (NZP + T64_RUN - 1) / T64_RUN;  // 33: 32 full runs and the last point

// v of either sign as a pair; 0 below 2^-70
__device__ __forceinline__ FF px_split_s(double v) {
  const double u = fabs(v);
  if (u < 8.5e-22) return FF{0.f, 0.f};
  const FF a = px_split(u);
  return v < 0.0 ? FF{-a.hi, -a.lo} : a;
}
// v 2^(1023 - ex) as a pair, ex the largest exponent field of the row; 0 where
// it is below 2^-70 of the row's largest
__device__ __forceinline__ FF px_split_scaled(double v, int ex) {
  const int h = __double2hiint(v), f = (h >> 20) & 0x7ff;
  if (f <= ex - 70 || f == 0) return FF{0.f, 0.f};
  return px_split_s(__hiloint2double(h + ((1023 - ex) << 20), __double2loint(v)));
}
__device__ __forceinline__ int exp_field(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// chi_x - chi of the node, chi = chi_w + sdw on its own segment, from three-float
// table values: far above a bin's redshift the points next to the node are the
// integral, and a rounding of chi would be 1e-13 of their differences
struct WlNode {
  F3 cw;
  FF sdw;
};
__device__ __forceinline__ FF wl_base(float2 cx, float cll, const WlNode& w) {
  const FF d = px_two_sum(cx.x, -w.cw.hi);
  return px_add(px_two_sum(d.hi, d.lo + ((cx.y - w.cw.lo) + (cll - w.cw.ll))), FF{-w.sdw.hi, -w.sdw.lo});
}

}  // namespace jcg
