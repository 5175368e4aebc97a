// rg_mul.cuh -- correctly rounded FP64 multiplication on the integer pipes.
//
// GB300 issues 1.75 FP64 operations per clock per SM (a warp instruction takes
// its sub-partition's FP64 unit for 64 clocks and four issue slots) and leaves
// the integer pipes of the FP64 kernels mostly idle.  mul_rn(a, b) returns the
// same bits as a * b (round to nearest even) for every pair of doubles in
// about 38 32-bit integer instructions, four of them 32 x 32 -> 64-bit
// multiply-adds, which keeps the ALU for about 50 clocks: less than the FP64
// unit's 64, and beside it.  A kernel bound by the FP64 unit forms some of its
// products here, up to where both pipes are equally busy.
//
// Method: the 53-bit significands as integers, Ma shifted to the top of a
// 64-bit word and Mb by one bit, so that the high word of their 128-bit product
// holds 53 or 54 significant bits; shifted to 54 bits, the lowest of them is
// the rounding bit.  Adding one unit of it where a lower bit of the product or
// the last kept bit is set, and dropping it, rounds to nearest even; a carry
// out of the significand raises the exponent field it is added to.  Zeros,
// subnormals, infinities, NaNs and products near the ends of the exponent
// range take a * b itself.
//
// tests/test_mul.py checks the host build against the host's product and the
// device build against the device's.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define RG_MUL_FN __host__ __device__ __forceinline__
#else
#define RG_MUL_FN inline
#endif

namespace rg {
namespace mul_detail {

RG_MUL_FN void words(double x, uint32_t& hi, uint32_t& lo) {
#if defined(__CUDA_ARCH__)
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
#else
  uint64_t u;
  std::memcpy(&u, &x, sizeof u);
  hi = static_cast<uint32_t>(u >> 32);
  lo = static_cast<uint32_t>(u);
#endif
}
RG_MUL_FN double assemble(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
#else
  const uint64_t u = (static_cast<uint64_t>(hi) << 32) | lo;
  double x;
  std::memcpy(&x, &u, sizeof x);
  return x;
#endif
}
// the high word of (hi:lo) << n, 0 <= n < 32
RG_MUL_FN uint32_t funnel_l(uint32_t lo, uint32_t hi, uint32_t n) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, n);
#else
  return n == 0 ? hi : (hi << n) | (lo >> (32 - n));
#endif
}

}  // namespace mul_detail

// A factor unpacked once for several products.
struct MulFactor {
  uint32_t top, bot;  // the 53-bit significand at the top of 64 bits
  uint32_t hi;        // the double's high word (sign, exponent)
};
RG_MUL_FN MulFactor mul_factor(double a) {
  uint32_t hi, lo;
  mul_detail::words(a, hi, lo);
  return MulFactor{mul_detail::funnel_l(lo, hi, 11) | 0x80000000u, lo << 11, hi};
}

// a * b on the fast path; returns false where the operands or the product are
// outside it (*p is then meaningless).
RG_MUL_FN bool mul_rn_fast(const MulFactor& a, double b, double* p) {
  using namespace mul_detail;
  uint32_t bhi, blo;
  words(b, bhi, blo);
  const uint32_t ea = a.hi & 0x7ff00000u, eb = bhi & 0x7ff00000u, es = ea + eb;
  // both normal, and the product's exponent field (es - 1023, in these units)
  // in [1, 2044]
  const bool ok = ea - 0x00100000u < 0x7fe00000u && eb - 0x00100000u < 0x7fe00000u && es - 0x40000000u < 0x7fd00000u;
  const uint32_t b1 = (funnel_l(blo, bhi, 1) & 0x001fffffu) | 0x00200000u, b0 = blo << 1;
  const uint64_t p0 = static_cast<uint64_t>(a.bot) * b0;
  const uint64_t p1 = static_cast<uint64_t>(a.top) * b0 + (p0 >> 32);
  const uint64_t p2 = static_cast<uint64_t>(a.bot) * b1 + static_cast<uint32_t>(p1);
  const uint64_t p3 = static_cast<uint64_t>(a.top) * b1 + ((p1 >> 32) + (p2 >> 32));
  const uint32_t h1 = static_cast<uint32_t>(p3 >> 32), h0 = static_cast<uint32_t>(p3);
  const uint32_t l1 = static_cast<uint32_t>(p2), l0 = static_cast<uint32_t>(p0);
  // p3 in [2^52, 2^54): to [2^53, 2^54)
  const bool wide = h1 >= 0x00200000u;
  const uint32_t s = wide ? 0u : 1u;
  const uint32_t t1 = funnel_l(h0, h1, s), t0 = funnel_l(l1, h0, s);
  // lower bits, or an odd last kept bit
  const uint32_t up = (l1 << s) | l0 | ((t0 >> 1) & 1u);
  const uint64_t t = ((static_cast<uint64_t>(t1) << 32) | t0) + (up != 0u ? 1u : 0u);
  // the hidden bit adds one to the exponent field
  const uint32_t r1 = static_cast<uint32_t>(t >> 33) + (es - (wide ? 0x3ff00000u : 0x40000000u));
  *p = assemble(r1 | ((a.hi ^ bhi) & 0x80000000u), static_cast<uint32_t>(t >> 1));
  return ok;
}
RG_MUL_FN bool mul_rn_fast(double a, double b, double* p) { return mul_rn_fast(mul_factor(a), b, p); }

#if defined(__CUDACC__)
// Products outside the fast path, out of line: inlined, the compiler
// predicates the FP64 instruction, and a predicated-off one still takes the
// unit's clocks.
static __device__ __noinline__ double mul_ieee(double a, double b) { return __dmul_rn(a, b); }
// (a zero and a finite operand, fluid at rest: formed without the FP64 unit)
static __device__ __noinline__ double mul_rest(double a, double b) {
  uint32_t ah, al, bh, bl;
  mul_detail::words(a, ah, al);
  mul_detail::words(b, bh, bl);
  const uint32_t am = ah & 0x7fffffffu, bm = bh & 0x7fffffffu;
  if (((am | al) == 0u || (bm | bl) == 0u) && am < 0x7ff00000u && bm < 0x7ff00000u)
    return mul_detail::assemble((ah ^ bh) & 0x80000000u, 0u);
  return mul_ieee(a, b);
}
// a * b, bitwise (fa: a unpacked)
__device__ __forceinline__ double mul_rn(const MulFactor& fa, double a, double b) {
  double p;
  if (!mul_rn_fast(fa, b, &p)) p = mul_rest(a, b);
  return p;
}
__device__ __forceinline__ double mul_rn(double a, double b) { return mul_rn(mul_factor(a), a, b); }
// a * x and a * y with one branch for both
__device__ __forceinline__ void mul_rn2(const MulFactor& fa, double a, double x, double y, double& ax, double& ay) {
  const bool ok0 = mul_rn_fast(fa, x, &ax), ok1 = mul_rn_fast(fa, y, &ay);
  if (!(ok0 && ok1)) {
    ax = mul_rest(a, x);
    ay = mul_rest(a, y);
  }
}
#endif

}  // namespace rg
