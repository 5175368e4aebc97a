// rg_trunc.cuh -- doubles truncated to floats on the integer pipe, for FP32
// estimates of FP64 decisions (rg_lgi.cuh, the CFL bounds, rg_3d.cu): three
// instructions and a range test where a rounding takes a dozen.
#pragma once
#include "rg_convert.cuh"

namespace rg {
namespace {

// x truncated to a float's 24 significant bits, on the integer pipe.  ok is
// cleared for a nonzero x outside the normal floats.
__device__ __forceinline__ float trunc32(double x, bool& ok) {
  const uint64_t u = conv_dbits(x);
  const uint32_t hi = static_cast<uint32_t>(u >> 32), lo = static_cast<uint32_t>(u);
  const uint32_t m = hi & 0x7fffffffu;
  // exponent field 897..1150 (0x381..0x47e)
  const bool in = m - 0x38100000u < 0x0fe00000u;
  ok = ok && (in || (m | lo) == 0u);
  const uint32_t t = __funnelshift_l(lo, hi, 3);
  return in ? __uint_as_float(((t ^ 0x40000000u) & 0x7fffffffu) | (hi & 0x80000000u)) : 0.0f;
}
// the same where a value below the normal floats may become 0 (an absolute
// error of 2^-126)
__device__ __forceinline__ float trunc32_any(double x, bool& ok) {
  const uint64_t u = conv_dbits(x);
  const uint32_t hi = static_cast<uint32_t>(u >> 32), lo = static_cast<uint32_t>(u);
  const uint32_t m = hi & 0x7fffffffu;
  ok = ok && m < 0x47f00000u;
  const uint32_t t = __funnelshift_l(lo, hi, 3);
  return m >= 0x38100000u ? __uint_as_float(((t ^ 0x40000000u) & 0x7fffffffu) | (hi & 0x80000000u)) : 0.0f;
}
// the same for a magnitude that only needs a lower bound: values below the
// normal floats become 0
__device__ __forceinline__ float trunc32_low(double x, bool& ok) {
  const uint64_t u = conv_dbits(x);
  const uint32_t hi = static_cast<uint32_t>(u >> 32), lo = static_cast<uint32_t>(u);
  const uint32_t m = hi & 0x7fffffffu;
  const bool in = m - 0x38100000u < 0x0fe00000u;
  ok = ok && m < 0x47f00000u;
  const uint32_t t = __funnelshift_l(lo, hi, 3);
  return in ? __uint_as_float((t ^ 0x40000000u) & 0x7fffffffu) : 0.0f;
}

}  // namespace
}  // namespace rg
