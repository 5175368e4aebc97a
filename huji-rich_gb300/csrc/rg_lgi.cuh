// rg_lgi.cuh -- LinearGaussImproved's slope and limiters for one component of
// one cell per thread (lane), shared by the hydro slopes (rg_fp64.cu, four
// lanes per cell) and the tracer slopes (rg_tracers.cu, one lane per tracer).
// Both units are compiled with --fmad=false.
//
// GB300 issues two FP64 operations per clock per SM against 64-128 FP32 or
// integer ones, so the limiter decides in FP32 which of a cell's centroid
// differences can set its factor psi, with a bound on the error of that
// decision, and forms only those in FP64, in the reference's operation order.
// psi is a minimum over the cell's faces, so leaving out a face whose
// candidate cannot be the minimum gives the same bits.
//
// Bounds.  With d = s_x dm_x + s_y dm_y in FP32 from s_x, s_y truncated to 24
// bits (2^-23 relative), dm rounded (2^-24) and two FP32 roundings, and
// A = |s_x dm_x| + |s_y dm_y|, d is within 3e-7 A of the real value; the
// FP64 difference fl(fl(fl(c + s_x dm_x) + s_y dm_y) - c) is within
// 2^-51 (|c| + A) of it.  E = 1e-6 A + 4e-15 |c| + 1e-36 covers both, the last
// term FP32 underflow of the products.  A slope outside the range of a normal
// float (and not zero), a |c| above it, or a centroid offset outside
// [1e-25, 1e25] (dm_screen stores NaN for it) makes every face a candidate.
#pragma once
#include "rg_adjoint.cuh"
#include "rg_fp64.cuh"
#include "rg_mul.cuh"
#include "rg_trunc.cuh"

namespace rg {
namespace {

constexpr int kFit = 8;  // neighbours held in registers; cells with more take the *_any forms

// A centroid offset as the screen reads it: NaN where the rounding to float
// would leave the range in which the bounds above hold.
__device__ __forceinline__ float dm_screen1(double v) {
  const uint64_t m = abs_u(v);
  if (m != 0u && !(m >= conv_dbits(1e-25) && m <= conv_dbits(1e25))) return __int_as_float(0x7fffffff);
  return narrow(v);
}
__device__ __forceinline__ float2 dm_screen(double2 dm) { return make_float2(dm_screen1(dm.x), dm_screen1(dm.y)); }

// a - b where only few warps need it: not computed ahead of its branch, as the
// compiler would (an FP64 operation costs a warp 16 clocks of the SM's pipe)
__device__ __forceinline__ double sub_here(double a, double b) {
  double r;
  asm volatile("sub.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}

// the double whose order_key is k (-0 becomes +0)
__device__ __forceinline__ double key_value(int64_t k) {
  return conv_double_bits(k < 0 ? static_cast<uint64_t>(-k) | 0x8000000000000000ull : static_cast<uint64_t>(k));
}

__device__ __forceinline__ double quad_value(unsigned quad, double v, int lane) {
  const uint64_t u = conv_dbits(v);
  const uint32_t lo = __shfl_sync(quad, static_cast<uint32_t>(u), lane, 4);
  const uint32_t hi = __shfl_sync(quad, static_cast<uint32_t>(u >> 32), lane, 4);
  return conv_double(hi, lo);
}

// Component q of a point's hydro state (point_state's): the value of the cell
// it copies, at(), and for the velocities of a rigid wall's ghosts the
// reflection, ghost().
struct HydroComp {
  const StepArgs& a;
  int q;
  __device__ __forceinline__ double at(int cell) const { return a.cells[4 * static_cast<size_t>(cell) + q]; }
  __device__ __forceinline__ bool reflects() const { return a.ghost_kind != RG_GHOST_PERIODIC && q >= 2; }
  __device__ __forceinline__ double ghost(int p, int cell, double v) const {
    const double2 u = a.geom.ghost_unit[p - a.mesh.n];
    const double2 vel = reinterpret_cast<const double2*>(a.cells)[2 * static_cast<size_t>(cell) + 1];
    const double s = 2 * (vel.x * u.x + vel.y * u.y);
    return v - (q == 2 ? u.x : u.y) * s;
  }
  __device__ __forceinline__ double operator()(int p) const {
    const int cell = copied_cell(a, p);
    const double v = at(cell);
    return p >= a.mesh.n && reflects() ? ghost(p, cell, v) : v;
  }
};
// Tracer j (a ghost carries the tracers of the cell it copies)
struct TracerComp {
  const StepArgs& a;
  const double* tr;
  int nt, j;
  __device__ __forceinline__ double at(int cell) const { return tr[static_cast<size_t>(cell) * nt + j]; }
  __device__ __forceinline__ bool reflects() const { return false; }
  __device__ __forceinline__ double ghost(int, int, double v) const { return v; }
  __device__ __forceinline__ double operator()(int p) const { return at(copied_cell(a, p)); }
};

// A cell's neighbours (at most kFit): values, and bit masks of the self-mirror
// ones and those that carry skip_key
struct LaneNeighbours {
  double v[kFit];
  unsigned mirror, skip;
};

template <class Load>
__device__ __forceinline__ void lane_load(const StepArgs& a, int b, int nn, const Load& load, LaneNeighbours& nb) {
  uint32_t w[kFit];
#pragma unroll
  for (int k = 0; k < kFit; ++k) w[k] = k < nn ? a.geom.nbr[b + k] : 0u;
  nb.mirror = nb.skip = 0u;
  unsigned ghosts = 0u;
#pragma unroll
  for (int k = 0; k < kFit; ++k) {
    const int p = static_cast<int>(w[k] & kNbrIdMask);
    nb.v[k] = 0.0;
    if (k < nn) nb.v[k] = load.at(copied_cell(a, p));
    nb.mirror |= (w[k] & kNbrMirror) ? 1u << k : 0u;
    ghosts |= p >= a.mesh.n ? 1u << k : 0u;
  }
  if (ghosts != 0u && load.reflects()) {
#pragma unroll
    for (int k = 0; k < kFit; ++k) {
      const int p = static_cast<int>(w[k] & kNbrIdMask);
      if ((ghosts >> k) & 1u) nb.v[k] = load.ghost(p, copied_cell(a, p), nb.v[k]);
    }
  }
  if (a.skip_mask != 0u) {
#pragma unroll
    for (int k = 0; k < kFit; ++k)
      if (k < nn && skipped(a, static_cast<int>(w[k] & kNbrIdMask))) nb.skip |= 1u << k;
  }
}

// The unlimited slope: :401-422 GetBoundarySlope or :80-133 calc_naive_slope.
__device__ __forceinline__ void lane_solve(const StepArgs& a, int i, bool boundary, double vx, double vy, double& sx,
                                           double& sy) {
  const dbl4 mi = a.geom.minv[i];
  if (boundary) {
    // vx, vy: sums of (neighbour - cell) * dx, dy; mi = {SxSy, Sx2, Sy2, den}
    sx = quot(vy * mi.x - vx * mi.z, mi.w);
    sy = quot(vx * mi.x - vy * mi.y, mi.w);
  } else {
    sx = vx * mi.x;
    sy = vy * mi.w;
    sx += vy * mi.y;
    sy += vx * mi.z;
  }
}
__device__ __forceinline__ void lane_slope(const StepArgs& a, int i, int b, int nn, bool boundary, double c,
                                           const LaneNeighbours& nb, double& sx, double& sy) {
  double vx = 0.0, vy = 0.0;
  if (boundary) {
#pragma unroll
    for (int k = 0; k < kFit; ++k) {
      if (k < nn) {
        const double2 h = a.geom.hr[b + k];
        const double df = sub_here(nb.v[k], c);
        vy = vy + df * h.y;
        vx = vx + df * h.x;
      }
    }
  } else {
    // the first neighbour starts the sums (cell*h, then + nb*h).  The cell's
    // products run on the integer pipes beside the FP64 unit (rg_mul.cuh):
    // 512^2 slopes 197 -> 172 us
    const MulFactor fc = mul_factor(c);
#pragma unroll
    for (int k = 0; k < kFit; ++k) {
      if (k < nn) {
        const double2 h = a.geom.hr[b + k];
        double cx, cy;
        mul_rn2(fc, c, h.x, h.y, cx, cy);
        if (k == 0) {
          vx = cx;
          vy = cy;
        } else {
          vx += cx;
          vy += cy;
        }
        vy += nb.v[k] * h.y;
        vx += nb.v[k] * h.x;
      }
    }
  }
  lane_solve(a, i, boundary, vx, vy, sx, sy);
}
template <class Load>
__device__ __forceinline__ void lane_slope_any(const StepArgs& a, int i, int b, int nn, bool boundary, double c,
                                               const Load& load, double& sx, double& sy) {
  double vx = 0.0, vy = 0.0;
  for (int k = 0; k < nn; ++k) {
    const double2 h = a.geom.hr[b + k];
    const double v = load(static_cast<int>(a.geom.nbr[b + k] & kNbrIdMask));
    if (boundary) {
      const double df = v - c;
      vy = vy + df * h.y;
      vx = vx + df * h.x;
    } else {
      if (k == 0) {
        vx = c * h.x;
        vy = c * h.y;
      } else {
        vx += c * h.x;
        vy += c * h.y;
      }
      vy += v * h.y;
      vx += v * h.x;
    }
  }
  lane_solve(a, i, boundary, vx, vy, sx, sy);
}

// What both forms of the limiter need of a cell: the extrema minus the cell,
// the 5 % / 10 % threshold, the dead band.
struct LaneRange {
  double maxd, mind, thr;
  int amax, amin;  // kTrace: the neighbour that gave the extremum, -1: the cell
};
__device__ __forceinline__ void lane_range(double c, int64_t kmax, int64_t kmin, bool shock, LaneRange& r) {
  r.maxd = key_value(kmax) - c;
  r.mind = key_value(kmin) - c;
  const double f = shock ? 0.1 : 0.05;
  r.thr = f * conv_double_bits(max_first_u(abs_u(r.maxd), abs_u(r.mind)));
}

// Face k's candidate in FP64 (:232-267 / :343-366), as limit_comp and
// shocked_comp take it; kTrace records the candidate that lowered psi.
template <bool kTrace, class Load>
__device__ __forceinline__ void lane_candidate(const StepArgs& a, int b, int k, double c, double sx, double sy,
                                               bool shock, bool abs_plain, bool abs_shock, const LaneRange& r,
                                               const Load& load, uint64_t& psi, float& psi_f, double& dphi_at,
                                               int& code) {
  const uint32_t w = a.geom.nbr[b + k];
  const double2 dm = centroid_offset(a.geom, w, a.mesh.cell_faces[b + k]);
  double cv = c;
  cv += sx * dm.x;
  cv += sy * dm.y;
  const double dphi = cv - c;
  const uint64_t before = psi;
  if (!shock) {
    limit_comp(dphi, cv, c, r.thr, r.maxd, r.mind, abs_plain, psi, psi_f);
    if (kTrace && psi != before) {
      // up where dphi > t1 (the upper dead-band threshold)
      const bool up = lt(abs_plain ? conv_double_bits(abs_u(1e-9 * c)) : 1e-9 * c, dphi);
      code = k | ((up ? 0 : 1) << 8) | (((up ? r.amax : r.amin) + 1) << 16);
      dphi_at = dphi;
    }
  } else {
    const double v = load(static_cast<int>(w & kNbrIdMask));
    shocked_comp(dphi, cv, c, r.thr, v, a.theta, psi, psi_f, abs_shock);
    if (kTrace && psi != before) {
      const bool clamp = quot(a.theta * (v - c), dphi) < 0.0;
      code = k | ((clamp ? 3 : 2) << 8) | ((k + 1) << 16);
      dphi_at = dphi;
    }
  }
}

// The limiter factor psi of a cell whose neighbours are in registers.
template <bool kTrace, class Load>
__device__ __forceinline__ void lane_limit(const StepArgs& a, int b, int nn, double c, double sx, double sy,
                                           bool shock, bool abs_plain, bool abs_shock, const LaneNeighbours& nb,
                                           const Load& load, double& psi_out, double& dphi_at, int& code) {
  // neighbour extrema as integer keys (std::max / std::min: the cell first);
  // the unshocked limiter skips self-mirror neighbours (:194-195), both the
  // skip_key ones (:192-193, :314-315)
  const unsigned out = nb.skip | (shock ? 0u : nb.mirror);
  int64_t kmax = order_key(conv_dbits(c)), kmin = kmax;
  LaneRange r;
  r.amax = r.amin = -1;
#pragma unroll
  for (int k = 0; k < kFit; ++k) {
    if (k < nn && !((out >> k) & 1u)) {
      const int64_t key = order_key(conv_dbits(nb.v[k]));
      if (kTrace && key > kmax) r.amax = k;
      if (kTrace && key < kmin) r.amin = k;
      kmax = key > kmax ? key : kmax;
      kmin = key < kmin ? key : kmin;
    }
  }
  lane_range(c, kmax, kmin, shock, r);
  // the FP32 screen
  bool ok = true;
  const float fx = trunc32(sx, ok), fy = trunc32(sy, ok);
  const float fc = trunc32_low(c, ok);
  const float fmax_ = trunc32_low(r.maxd, ok), fmin_ = trunc32_low(r.mind, ok);  // lower bounds of maxd, -mind
  float d[kFit];
  float big = 0.0f, dmax = -1e38f, dmin = 1e38f;
#pragma unroll
  for (int k = 0; k < kFit; ++k) {
    d[k] = 0.0f;
    if (k < nn) {
      const float2 m = a.geom.dmf[b + k];
      const float px = fx * m.x, py = fy * m.y;
      const float s = fabsf(px) + fabsf(py);
      d[k] = fmaf(fx, m.x, py);
      ok = ok && s < 1e37f;  // false for NaN
      big = fmaxf(big, s);
      dmax = fmaxf(dmax, d[k]);
      dmin = fminf(dmin, d[k]);
    }
  }
  const float err = fmaf(big, 1e-6f, fmaf(fc, 4e-15f, 1e-36f));
  const bool c_neg = (conv_dbits(c) >> 63) != 0u;
  // below the threshold and too small to change the sign: inactive
  const float thr_lo = (shock ? 0.1f : 0.05f) * fmaxf(fmax_, fmin_);
  const float idle = 0.99999f * fminf(thr_lo, fc);
  const float dead = 0.999e-9f * fc;
  unsigned mask = 0u;
  uint64_t psi = kOneBits;
  float psi_f = 1.0f;
  if (!shock) {
    // Of the faces above (below) the dead band the largest (smallest) dphi
    // gives the smallest candidate, and it is active if any of them is: with
    // one sign of dphi the quotient, |dphi| > thr and the sign change of
    // cv = c + dphi are all monotone in it.  So psi stays 1 when neither
    // extreme can overshoot the neighbours' range (or both are inactive), and
    // otherwise only faces within 2 E of an extreme are formed.
    const float lim = fmaxf(dead, idle);
    const bool up = !(dmax + err <= fmaxf(fmax_, lim)), down = !(err - dmin <= fmaxf(fmin_, lim));
    const float hi = up ? dmax - 2.0f * err : 3e38f, lo = down ? dmin + 2.0f * err : -3e38f;
#pragma unroll
    for (int k = 0; k < kFit; ++k)
      if (k < nn && (d[k] >= hi || d[k] <= lo)) mask |= 1u << k;
    // a negative value without the absolute value has a dead band of the
    // other sign; a zero numerator ties every candidate (the trace keeps the first)
    ok = ok && (abs_plain || !c_neg) && (!kTrace || (fmax_ > 0.0f && fmin_ > 0.0f));
    if (!ok) mask = (1u << nn) - 1u;
  } else {
    // the candidates max(theta (nb - c) / dphi, 0) differ in their
    // numerators: a lower bound for each face, an upper bound of the minimum
    float low[kFit];
    float best = 1.0f;
    const float th = trunc32(a.theta, ok);
    const float thr_hi = 1.00001f * thr_lo, dead_hi = 1.001e-9f * fc;
    const float dead_s = abs_shock || !c_neg ? dead : -1.0f;
    ok = ok && th > 1e-6f && th < 1e6f;
    bool ok_nb = true;
#pragma unroll
    for (int k = 0; k < kFit; ++k) {
      low[k] = 3e38f;
      if (k < nn && !((nb.skip >> k) & 1u)) {
        const float ad = fabsf(d[k]);
        if (!(ad + err <= idle || ad + err <= dead_s)) {
          low[k] = 0.0f;
          // the FP64 difference: neighbours often agree to more bits than a float has
          const float g = trunc32(sub_here(nb.v[k], c), ok_nb);
          if (ok_nb && ad - err > thr_hi && ad - err > dead_hi && fabsf(g) > 1e-30f) {
            if ((g < 0.0f) != (d[k] < 0.0f)) {
              best = 0.0f;  // the candidate is 0
            } else {
              const float q = __fdividef(th * fabsf(g), ad);
              const float rel = 2e-6f + 2.0f * __fdividef(err, ad);
              // (below the normal floats q's error is absolute: formed in FP64)
              if (rel < 0.1f && q > 1e-30f) {
                low[k] = q * (1.0f - rel);
                best = fminf(best, q * (1.0f + rel));
              }
            }
          }
        }
      }
    }
    ok = ok && ok_nb;
#pragma unroll
    for (int k = 0; k < kFit; ++k)
      if (low[k] <= best) mask |= 1u << k;
    if (!ok) {
      mask = ((1u << nn) - 1u) & ~nb.skip;
    } else if (!kTrace && best == 0.0f) {
      psi = 0u;
      mask = 0u;
    }
  }
  // a zero slope: every dphi is 0 (or NaN), which no candidate takes
  if (((conv_dbits(sx) | conv_dbits(sy)) & kMagMask) == 0u) {
    mask = 0u;
    psi = kOneBits;
  }
  while (mask) {
    const int k = __ffs(mask) - 1;
    mask &= mask - 1u;
    lane_candidate<kTrace>(a, b, k, c, sx, sy, shock, abs_plain, abs_shock, r, load, psi, psi_f, dphi_at, code);
  }
  psi_out = conv_double_bits(psi);
}

// The same for any number of neighbours: every face's candidate in FP64.
template <bool kTrace, class Load>
__device__ __forceinline__ void lane_limit_any(const StepArgs& a, int b, int nn, double c, double sx, double sy,
                                               bool shock, bool abs_plain, bool abs_shock, const Load& load,
                                               double& psi_out, double& dphi_at, int& code) {
  int64_t kmax = order_key(conv_dbits(c)), kmin = kmax;
  LaneRange r;
  r.amax = r.amin = -1;
  for (int k = 0; k < nn; ++k) {
    const uint32_t w = a.geom.nbr[b + k];
    const int p = static_cast<int>(w & kNbrIdMask);
    if ((!shock && (w & kNbrMirror)) || skipped(a, p)) continue;
    const int64_t key = order_key(conv_dbits(load(p)));
    if (key > kmax) {
      kmax = key;
      r.amax = k;
    }
    if (key < kmin) {
      kmin = key;
      r.amin = k;
    }
  }
  lane_range(c, kmax, kmin, shock, r);
  uint64_t psi = kOneBits;
  float psi_f = 1.0f;
  for (int k = 0; k < nn; ++k) {
    if (shock && skipped(a, static_cast<int>(a.geom.nbr[b + k] & kNbrIdMask))) continue;  // :339-340
    lane_candidate<kTrace>(a, b, k, c, sx, sy, shock, abs_plain, abs_shock, r, load, psi, psi_f, dphi_at, code);
  }
  psi_out = conv_double_bits(psi);
}

}  // namespace
}  // namespace rg
