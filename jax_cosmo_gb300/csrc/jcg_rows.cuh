// What the halofit rows of both precisions share.
#pragma once

#include "jcg_internal.cuh"

namespace jcg {

constexpr double TWO_PI2 = 2.0 * (PI * PI);  // 2.0 * np.pi**2
constexpr double C2 = C_KMS * C_KMS;          // const.c**2

struct HfParams {
  double knl, neff, C;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// chi at a from the table (background.py:242) with the segment chosen by the
// reference's rule and the precomputed slopes
__device__ __forceinline__ double chi_at(const CosmoTab* ct, const ConstTables* c, double a, int2 seg) {
  const int k = min(seg.x, seg.y);
  return fmax(ct->chi[seg.x] + ct->chi_slope[k] * (a - c->atab_chi[seg.x]), 0.0);
}

}  // namespace jcg
