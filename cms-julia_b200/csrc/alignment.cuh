// The alignment cut of the connection test and its bound; host-callable, so that the bound is checked on the CPU
// (built there without contraction: every operation is rounded by itself).
#pragma once
#include <cmath>

#define PXL_HD __host__ __device__ __forceinline__

namespace pxl {

// CA parameters (ca_hit_ntuplet_generator.jl:9-30), Float32 as Params stores them
constexpr float kPtMin = 0.899999976158f;
constexpr float kThetaBarrel = 0.00200000009499f;
constexpr float kThetaForward = 0.00300000002608f;

#ifdef __CUDA_ARCH__
PXL_HD float add_rn(float a, float b) { return __fadd_rn(a, b); }
PXL_HD float sub_rn(float a, float b) { return __fsub_rn(a, b); }
PXL_HD float mul_rn(float a, float b) { return __fmul_rn(a, b); }
PXL_HD float sqrt_rn(float a) { return __fsqrt_rn(a); }
PXL_HD float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
#else
PXL_HD float add_rn(float a, float b) { return a + b; }
PXL_HD float sub_rn(float a, float b) { return a - b; }
PXL_HD float mul_rn(float a, float b) { return a * b; }
PXL_HD float sqrt_rn(float a) { return sqrtf(a); }
PXL_HD float fma_rn(float a, float b, float c) { return fmaf(a, b, c); }
#endif

PXL_HD bool are_aligned(float r1, float z1, float ri, float zi, float ro, float zo, float theta_cut) {
  const float radius_diff = fabsf(sub_rn(r1, ro));
  const float dz = sub_rn(z1, zo);
  const float d13 = add_rn(mul_rn(radius_diff, radius_diff), mul_rn(dz, dz));
  const float p_min = mul_rn(kPtMin, sqrt_rn(d13));
  const float t = fabsf(add_rn(add_rn(mul_rn(z1, sub_rn(ri, ro)), mul_rn(zi, sub_rn(ro, r1))), mul_rn(zo, sub_rn(r1, ri))));
  return mul_rn(t, p_min) <= mul_rn(mul_rn(theta_cut, d13), radius_diff);
}

// False only where are_aligned is false, without its square root: the two sides squared, the right one
// larger by a share that covers the rounding of both (1e-6) and by a term above all underflow.
PXL_HD bool maybe_aligned(float r1, float z1, float ri, float zi, float ro, float zo, bool barrel) {
  constexpr float kBarrel = float(double(kThetaBarrel) * kThetaBarrel / (0.899999976158 * 0.899999976158) * (1 + 1e-5));
  constexpr float kForward = float(double(kThetaForward) * kThetaForward / (0.899999976158 * 0.899999976158) * (1 + 1e-5));
  const float u = sub_rn(ro, r1);
  const float t = add_rn(add_rn(mul_rn(z1, sub_rn(ri, ro)), mul_rn(zi, u)), mul_rn(zo, sub_rn(r1, ri)));
  const float dz = sub_rn(z1, zo), u2 = mul_rn(u, u);
  const float lim = fma_rn(mul_rn(u2, fma_rn(dz, dz, u2)), barrel ? kBarrel : kForward, 1e-30f);
  return !(mul_rn(t, t) > lim);
}

}  // namespace pxl
