// rg_face.cuh -- Hllc in FP64 for the per-face kernels, with as little of it on
// the FP64 unit as the bits allow: the same operations on the same operands as
// hllc() in rg_hllc.cuh (and so the reference's), in straight-line code.
//
// GB300's FP64 unit takes 64 clocks of an SM sub-partition per warp
// instruction.  What moved off it, or out of the kernel:
//   * comparisons and the tests for NaN run on the operands' bit patterns;
//   * quotients by one divisor share its preparation (rg_div.cuh);
//   * quantities that only the upwind side needs (internal energy, tangential
//     velocity, kinetic energy) are formed for that side alone;
//   * a good half of the products run on the integer pipes (rg_mul.cuh).
// Operands outside the integer forms' range (subnormals, infinities, NaN, an
// invalid solution) clear `ok`; the caller then solves the face by hllc().
#pragma once
#include "rg_convert.cuh"
#include "rg_div.cuh"
#include "rg_hllc.cuh"
#include "rg_mul.cuh"

namespace rg {
namespace {

struct FaceOps {
  bool ok = true;
  __device__ __forceinline__ Divisor by(double b) {
    const Divisor D = divisor(b, RcpSeedDevice{});
    ok = ok && D.ok;
    return D;
  }
  __device__ __forceinline__ double div(double a, const Divisor& D) {
    double q;
    ok = div_by(a, D, &q) && ok;
    return q;
  }
  __device__ __forceinline__ double sqrt(double x) {
    double r;
    ok = sqrt_rn_fast(x, RsqrtSeedDevice{}, &r) && ok;
    return r;
  }
  // a product on the integer pipes; the FP64 unit's where it is outside them
  // (zeros above all)
  __device__ __forceinline__ double mul(double a, double b) { return mul_rn(a, b); }
};

__device__ __forceinline__ uint32_t hi_word(double x) {
  uint32_t hi, lo;
  mul_detail::words(x, hi, lo);
  return hi;
}
// |hi| of a double for the test x is infinite or NaN: >= 0x7ff00000
__device__ __forceinline__ uint32_t mag_hi(double x) { return hi_word(x) & 0x7fffffffu; }
__device__ __forceinline__ bool is_zero(double x) { return (conv_dbits(x) & kMagMask) == 0u; }
__device__ __forceinline__ bool sign_bit(double x) { return (hi_word(x) >> 31) != 0u; }
// a < b for finite a, b (order of the bit patterns; -0 below +0)
__device__ __forceinline__ bool less_finite(double a, double b) {
  const int64_t x = static_cast<int64_t>(conv_dbits(a)), y = static_cast<int64_t>(conv_dbits(b));
  return (x ^ static_cast<int64_t>(static_cast<uint64_t>(x >> 63) >> 1)) <
         (y ^ static_cast<int64_t>(static_cast<uint64_t>(y >> 63) >> 1));
}
// 0.5 * x, on the exponent where that is all it changes
__device__ __forceinline__ double half_of(double x) {
  const uint64_t u = conv_dbits(x);
  const uint32_t m = static_cast<uint32_t>(u >> 32) & 0x7fffffffu;
  double r = x;
  if (m - 0x00200000u < 0x7fd00000u)
    r = conv_double_bits(u - 0x0010000000000000ull);
  else if ((u & kMagMask) != 0u)
    r = mul_ieee(0.5, x);
  return r;
}
__device__ __forceinline__ Divisor pick(bool first, const Divisor& a, const Divisor& b) {
  return Divisor{first ? a.mb : b.mb, first ? a.R1 : b.R1, first ? a.r0 : b.r0, first ? a.eb : b.eb,
                 first ? a.sign : b.sign, first ? a.ok : b.ok};
}

struct FaceSide {
  double d, p, vx;  // density, pressure, normal velocity
};

// hllc() (hllc.cpp:97-154) of two sides in the face frame.  vy(left): that
// side's tangential velocity; velocity: the face's normal speed (moving: not
// +-0); gm1: gamma - 1.  left tells which side the flux is formed from.
template <class Vy>
__device__ __forceinline__ void hllc_face(FaceOps& o, FaceSide l, FaceSide r, double g, const Divisor& gm1,
                                          bool moving, double velocity, const Vy& vy, Cons& f, bool& left) {
  const Divisor dl = o.by(l.d), dr = o.by(r.d);
  const double cl = o.sqrt(o.div(o.mul(g, l.p), dl)), cr = o.sqrt(o.div(o.mul(g, r.p), dr));
  if (moving) {
    l.vx -= velocity;
    r.vx -= velocity;
  }
  // :27-43 estimate_wave_speeds
  const double a1 = l.vx - cl, b1 = r.vx - cr, a2 = l.vx + cl, b2 = r.vx + cr;
  const double sl = less_finite(b1, a1) ? b1 : a1;
  const double sr = less_finite(a2, b2) ? b2 : a2;
  const double tl = sl - l.vx, tr = sr - r.vx;
  const double ss = o.div(r.p - l.p + o.mul(o.mul(l.d, l.vx), tl) - o.mul(o.mul(r.d, r.vx), tr),
                          o.by(o.mul(l.d, tl) - o.mul(r.d, tr)));
  // finite wave speeds: the left side applies where sl > 0 or the contact does
  // not move left, the right side otherwise
  uint32_t top = max(max(mag_hi(a1), mag_hi(b1)), max(mag_hi(a2), mag_hi(b2)));
  top = max(top, mag_hi(ss));
  o.ok = o.ok && top < 0x7ff00000u;
  const bool slpos = !sign_bit(sl) && !is_zero(sl), srneg = sign_bit(sr) && !is_zero(sr);
  const bool ssneg = sign_bit(ss) && !is_zero(ss);
  left = slpos || !ssneg;
  const double d = left ? l.d : r.d, p = left ? l.p : r.p, vx = left ? l.vx : r.vx, sk = left ? sl : sr;
  const Divisor D = pick(left, dl, dr);
  const double vt = vy(left);
  // ideal_gas.cpp:13-16, hydrodynamic_variables.cpp:261-265
  const double pd = o.div(p, D), e = o.div(pd, gm1);
  const double s = o.sqrt(o.mul(vx, vx) + o.mul(vt, vt));
  const double ek = d * (half_of(o.mul(s, s)) + e);
  const double dsp = o.mul(d, vx);
  // :281-290 Primitive2Flux along (1,0)
  Cons fk{dsp, p + o.mul(vx, dsp), o.mul(vt, dsp), (ek + p) * vx};
  if (left ? !slpos : !srneg) {
    // :76-92 starred_state
    const double skv = sk - vx;
    const double ds = o.div(o.mul(d, skv), o.by(sk - ss));
    const double use = o.div(o.mul(ek, ds), D) + o.mul(o.mul(ds, ss - vx), ss + o.div(pd, o.by(skv)));
    fk.m = fk.m + sk * (ds - d);
    fk.mx = fk.mx + (o.mul(ds, ss) - dsp) * sk;
    fk.my = fk.my + (o.mul(ds, vt) - o.mul(vt, d)) * sk;
    fk.en = fk.en + sk * (use - ek);
  }
  // :150-152 back to the lab frame along the normal
  if (moving) {
    fk.en += fk.mx * velocity + half_of(fk.m) * velocity * velocity;
    fk.mx += velocity * fk.m;
  }
  f = fk;
}

}  // namespace
}  // namespace rg
