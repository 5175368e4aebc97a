// rg_limit32.cuh -- LinearGaussImproved's limiters of one component in FP32
// (LinearGaussImproved.cpp:174-399), shared by the FP32-mixed slopes kernels.
#pragma once
#include <cuda_runtime.h>

namespace rg {
namespace {

// The limiters' candidate of one neighbour, without branches: the candidate
// quotient is always formed and taken only where the limiter takes it, so
// psi is the same bits as with the limiter's if / else-if, and a warp's
// lanes never diverge here.
__device__ __forceinline__ void limit32(float dphi, float cv, float cellv, float thr, float maxd, float mind,
                                        bool use_abs, float& psi) {
  const bool active = fabsf(dphi) > thr || cv * cellv < 0.0f;
  const float t = use_abs ? fabsf(1e-9f * cellv) : 1e-9f * cellv;
  const float nt = use_abs ? -fabsf(1e-9f * cellv) : -1e-9f * cellv;
  const bool up = dphi > t;
  const float cand = __fdividef(up ? maxd : mind, dphi);
  psi = active && (up || dphi < nt) ? fminf(psi, cand) : psi;
}

__device__ __forceinline__ void shocked32(float dphi, float cv, float cellv, float thr, float nbv, float theta,
                                          float& psi) {
  const bool active = (fabsf(dphi) > thr || cv * cellv < 0.0f) && fabsf(dphi) > 1e-9f * cellv;
  const float cand = fmaxf(__fdividef(theta * (nbv - cellv), dphi), 0.0f);
  psi = active ? fminf(psi, cand) : psi;
}

// The unshocked limiter of one component from the largest and the smallest
// reconstructed value over the cell's faces: among the faces with a positive
// centroid difference the largest has the smallest quotient maxd/dphi (the
// FP32 quotient is monotone in its divisor, checked over every positive divisor
// for eight numerators: tests/limit32_check.cu),
// and it is active if any of them is, as |dphi| and the change of sign only
// grow with it; with mind the smallest of the negative ones likewise.  psi is
// their minimum, so no other face can set it.
__device__ __forceinline__ float limit32_range(float hi, float lo, float cellv, float thr, float maxd, float mind,
                                               bool use_abs) {
  float psi = 1.0f;
  limit32(hi - cellv, hi, cellv, thr, maxd, __int_as_float(0x7fffffff), use_abs, psi);
  limit32(lo - cellv, lo, cellv, thr, __int_as_float(0x7fffffff), mind, use_abs, psi);
  return psi;
}

}  // namespace
}  // namespace rg
