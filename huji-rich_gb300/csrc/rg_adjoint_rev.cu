// rg_adjoint_rev.cu -- hand-written reverse sweep of one differentiated step
// (FP64; rg_adjoint_rev32.cu builds the face and cell kernels again in FP32
// for the FP32-mixed adjoint).  With Ubar_{k+1} = dL/dU_{k+1} given, one reverse step is
//     Wbar_k = G'(W_k)^T Ubar_{k+1}
//     Ubar_k = Ubar_{k+1} + C'(U_k)^T Wbar_k      (k > 0)
//     dL/dW_0 = Wbar_0 + I'(W_0)^T Ubar_1          (k = 0)
// and G'^T runs as three kernels, each a gather with no atomics:
//   k_adj_faces  per face: the flux adjoint dt*area*(Ubar[second] -
//                Ubar[first]) (the transposed SimpleExtensiveUpdater
//                gather) through the rotation back, HLLC (the primal's wave
//                speed and region branches) and the rotation into the face
//                frame, to the adjoints of the face's two reconstructed states
//   k_adj_cell   per cell: gathers the adjoints of the face states built
//                from it (its own sides and those of the periodic ghosts it
//                is the source of) into its state and slope adjoints, then
//                reverses the limiter (the active candidate in the trace:
//                psi = numerator/dphi, a subgradient at switches) and the
//                Green-Gauss slope; the shares of its neighbours are written
//                per CSR entry
//   k_adj_update gathers the CSR-entry shares addressed to the cell (the
//                reverse adjacency, ascending), adds its own share and
//                applies C'^T (or I'^T for the first step)
// The branches are re-evaluated from the stored forward state; this file
// lets the compiler contract multiply-adds, so a re-evaluation can differ
// from the forward only at an exact tie, where either side is a valid
// one-sided derivative.
#include <math.h>

#include "rg_launch.cuh"
#include "rg_adjoint.cuh"
#include "rg_div.cuh"
#include "rg_face.cuh"

#ifndef RG_ADJ_REAL
#define RG_ADJ_REAL double
#define RG_ADJ_FP64 1
#endif

namespace rg {
namespace {

// (per cell: small blocks spread a 256^2 mesh's 1 to 4 warps per SM sub-partition
// evenly; cells 34.9 us in blocks of 256, 33.5 of 64, update 12.7 and 12.1)
constexpr int kBlock = 64;
constexpr int kFaceBlock = 128;  // k_adj_faces

__device__ __forceinline__ void load_raw(const double* c, int i, double o[4]) {
  const double2 a = reinterpret_cast<const double2*>(c)[2 * i];
  const double2 b = reinterpret_cast<const double2*>(c)[2 * i + 1];
  o[0] = a.x;
  o[1] = a.y;
  o[2] = b.x;
  o[3] = b.y;
}
__device__ __forceinline__ void store_raw(double* c, int i, const double v[4]) {
  reinterpret_cast<double2*>(c)[2 * i] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(c)[2 * i + 1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ int source_of(const MeshDev& m, int p) { return p < m.n ? p : m.ghost_source[p - m.n]; }

// Working precision of the face and cell reverse kernels: double here;
// rg_adjoint_rev32.cu compiles them again with float (the FP32-mixed
// adjoint).  The recorded steps and the arrays between the kernels are of the
// same precision (kept in FP64, the FP32 faces took 26 us where they take 16,
// the trace slopes 18 where they take 15, at 256^2).
using real = RG_ADJ_REAL;
struct rv2 {
  real x, y;
};
__device__ __forceinline__ real to_real(double x) {
#if RG_ADJ_FP64
  return x;
#else
  return narrow(x);
#endif
}
#if RG_ADJ_FP64
using Trace = SlopeTrace;
__device__ __forceinline__ void load_r(const void* c, int i, real o[4]) { load_raw(static_cast<const double*>(c), i, o); }
__device__ __forceinline__ void store_r(void* c, int i, const real v[4]) { store_raw(static_cast<double*>(c), i, v); }
__device__ __forceinline__ void load_wide(const void* c, int i, double o[4]) { load_r(c, i, o); }
// the geometry
__device__ __forceinline__ rv2 r2(double2 v) { return rv2{v.x, v.y}; }
__device__ __forceinline__ rv2 side_dm(const AdjArgs& a, int e, bool first) {
  return r2(first ? a.geom.dm0[e] : a.geom.dm1[e]);
}
__device__ __forceinline__ rv2 entry_dm(const AdjArgs& a, int k) {
  return side_dm(a, a.mesh.cell_faces[k], a.geom.nbr[k] & kNbrFirst);
}
__device__ __forceinline__ rv2 entry_h(const AdjArgs& a, int k) { return r2(a.geom.hr[k]); }
__device__ __forceinline__ void load_minv(const AdjArgs& a, int i, real mi[4]) {
  const dbl4 v = a.geom.minv[i];
  mi[0] = v.x, mi[1] = v.y, mi[2] = v.z, mi[3] = v.w;
}
#else
using Trace = SlopeTrace32;
__device__ __forceinline__ void load_r(const void* c, int i, real o[4]) {
  const float4 v = static_cast<const float4*>(c)[i];
  o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
}
__device__ __forceinline__ void store_r(void* c, int i, const real v[4]) {
  static_cast<float4*>(c)[i] = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void load_wide(const void* c, int i, double o[4]) {
  real v[4];
  load_r(c, i, v);
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = widen_exact(v[q]);
}
// the geometry: the handle's FP32 copies (roundings of the FP64 arrays)
__device__ __forceinline__ rv2 r2(float2 v) { return rv2{v.x, v.y}; }
__device__ __forceinline__ rv2 side_dm(const AdjArgs& a, int e, bool first) {
  return r2(first ? a.g32.dm0[e] : a.g32.dm1[e]);
}
__device__ __forceinline__ rv2 entry_dm(const AdjArgs& a, int k) {
  const float4 v = a.g32.ent[k];
  return rv2{v.z, v.w};
}
__device__ __forceinline__ rv2 entry_h(const AdjArgs& a, int k) {
  return r2(*reinterpret_cast<const float2*>(a.g32.ent + k));
}
__device__ __forceinline__ void load_minv(const AdjArgs& a, int i, real mi[4]) {
  const float4 v = a.g32.minv[i];
  mi[0] = v.x, mi[1] = v.y, mi[2] = v.z, mi[3] = v.w;
}
#endif

// C'(U)^T w for SimpleCellUpdater (d = m/V, v = P/m, e = E/m - |v|^2/2,
// p = (gamma-1) e d), added to ub.
__device__ __forceinline__ void cell_update_transpose(double gamma, double V, const double u[4], const double w[4],
                                                      double ub[4]) {
  const double mass = u[0], en = u[1];
  const double d = quot(mass, V), vx = quot(u[2], mass), vy = quot(u[3], mass);
  const double e = quot(en, mass) - 0.5 * (vx * vx + vy * vy);
  const double be = w[1] * (gamma - 1) * d;
  const double bd = w[0] + w[1] * (gamma - 1) * e;
  const double bvx = w[2] - be * vx, bvy = w[3] - be * vy;
  ub[0] += quot(bd, V) - quot(quot(be * en, mass) + bvx * vx + bvy * vy, mass);
  ub[1] += quot(be, mass);
  ub[2] += quot(bvx, mass);
  ub[3] += quot(bvy, mass);
}

#if RG_ADJ_FP64
// Periodic meshes only: every ghost has a source, no CSR entry is a
// self-mirror and no cell uses the boundary slope.
__global__ void __launch_bounds__(kBlock) k_adj_check(AdjArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < a.mesh.m && (a.geom.nbr[t] & kNbrMirror)) record_error(a.status, 0, RG_ERR_INVALID_ARGUMENT, 0, t, 0.0);
  if (t < a.mesh.n && (a.geom.cflags[t] & kCellBoundarySlope))
    record_error(a.status, 0, RG_ERR_INVALID_ARGUMENT, 1, t, 0.0);
}

__global__ void __launch_bounds__(kBlock) k_adj_seed(AdjArgs a, const double* wbar, double* ubar) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.mesh.n) return;
  double u[4], w[4], ub[4] = {0, 0, 0, 0};
  load_raw(a.ext, i, u);
  load_raw(wbar, i, w);
  cell_update_transpose(a.gamma, a.mesh.cd_volume[i], u, w, ub);
  store_raw(ubar, i, ub);
}

#endif  // RG_ADJ_FP64

#if RG_ADJ_FP64
template <class O>
__device__ __forceinline__ double scaled(O& o, double x, double s) { return o.mul(x, s); }
#else
__device__ __forceinline__ double scaled(int&, double x, double s) { return x * s; }
#endif

#if RG_ADJ_FP64
// The operations of the reverse in plain arithmetic, for operands outside the
// integer forms' range (FaceOps clears ok there).
struct PlainOps {
  static constexpr bool ok = true;
  __device__ __forceinline__ double by(double b) { return b; }
  __device__ __forceinline__ double by(const Divisor&, double b) { return b; }
  __device__ __forceinline__ double div(double a, double b) { return a / b; }
  __device__ __forceinline__ double sqrt(double x) { return ::sqrt(x); }
  __device__ __forceinline__ double mul(double a, double b) { return a * b; }
  __device__ __forceinline__ double half(double x) { return 0.5 * x; }
  __device__ __forceinline__ void finite(double, double, double, double) {}
  static __device__ __forceinline__ double pick(bool first, double a, double b) { return first ? a : b; }
};
struct RevOps : FaceOps {
  using FaceOps::by;
  __device__ __forceinline__ Divisor by(const Divisor& D, double) {
    ok = ok && D.ok;
    return D;
  }
  __device__ __forceinline__ double half(double x) { return half_of(x); }
  __device__ __forceinline__ void finite(double a, double b, double c, double d) {
    ok = ok && max(max(mag_hi(a), mag_hi(b)), max(mag_hi(c), mag_hi(d))) < 0x7ff00000u;
  }
  static __device__ __forceinline__ Divisor pick(bool first, const Divisor& a, const Divisor& b) {
    return rg::pick(first, a, b);
  }
};
__device__ __forceinline__ bool positive(double x) { return !sign_bit(x) && !is_zero(x); }
__device__ __forceinline__ bool negative(double x) { return sign_bit(x) && !is_zero(x); }
// a + b where only few warps need it, not computed ahead of its branch
__device__ __forceinline__ double add_here(double a, double b) {
  double r;
  asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}

// Reverse of primitive conversion, rotation into the face frame, Hllc
// (hllc.cpp:97-154, massflux, face at rest) and the rotation back: from fb
// (adjoint of {mass, energy, px, py}) to the adjoints of the two states.
//
// Hllc's flux is written the way it is cheapest to reverse.  With J = d (S_K - u)
// the mass flux through the outer wave and z the contact speed S*, the flux
// F_K + S_K (U* - U_K) equals
//     {m, E' m + p* z, p* + m z, m v_t},   m = d* z,   d* = J/(S_K - z),
//     p* = p + J A,   E' = |v|^2/2 + e + A B,   A = z - u,   B = z + p/J,
// and the flux of an undisturbed side is the same with z = u, d* = d, p* = p, A = 0.
// The reverse of this form takes 80 FP64 additions or multiply-adds where the
// reverse of the former takes 240 FP64 operations, and is as accurate or
// better (20,000 random faces against 80-bit arithmetic: mean error 2.4e-16 of
// the largest adjoint against 4.3e-16, worst 3.1e-15 against 1.6e-14).
template <class O>
__device__ __forceinline__ void hllc_reverse(O& o, double g, const Divisor& gm1, rv2 n, double na, rv2 p, double pa,
                                             const double L[4], const double R[4], const double fb[4], double lb[4],
                                             double rb[4]) {
  // forward values
  const double dL = L[0], pL = L[1], dR = R[0], pR = R[1];
  const auto qdL = o.by(dL), qdR = o.by(dR), qna = o.by(na), qpa = o.by(pa), qgm1 = o.by(gm1, g - 1.0);
  const double cL = o.sqrt(o.div(o.mul(g, pL), qdL)), cR = o.sqrt(o.div(o.mul(g, pR), qdR));
  const double lu = o.div(o.mul(L[2], n.x) + L[3] * n.y, qna), ru = o.div(o.mul(R[2], n.x) + R[3] * n.y, qna);
  const double a1 = lu - cL, b1 = ru - cR, a2 = lu + cL, b2 = ru + cR;
  const bool sl_right = less_finite(b1, a1), sr_right = less_finite(a2, b2);
  const double sl = sl_right ? b1 : a1, sr = sr_right ? b2 : a2;
  o.finite(a1, b1, a2, b2);  // the tests on signs and bit patterns are for finite speeds
  const double tl = sl - lu, tr = sr - ru;
  const double JL = o.mul(dL, tl), JR = o.mul(dR, tr);
  const auto qden = o.by(JL - JR);
  const double ss = o.div((pR - pL) + JL * lu - JR * ru, qden);
  const bool left = positive(sl) || !negative(ss);
  const bool star = left ? !positive(sl) : !negative(sr);
  // the upwind side
  const double qd = left ? dL : dR, qp = left ? pL : pR, qu = left ? lu : ru, sk = left ? sl : sr;
  const double K = left ? tl : tr, J = left ? JL : JR;
  const auto by_d = O::pick(left, qdL, qdR);
  const double qv = o.div(o.mul(left ? L[2] : R[2], p.x) + (left ? L[3] : R[3]) * p.y, qpa);
  const double e = o.div(o.div(qp, by_d), qgm1);
  double E = 0.5 * (qu * qu + o.mul(qv, qv)) + e;
  // adjoint of the face-frame flux {fm, fmx, fmy, fen}
  const double bfm = fb[0], bfen = fb[1];
  const double bfmx = o.div(n.x * fb[2] + o.mul(n.y, fb[3]), qna);
  const double bfmy = o.div(p.x * fb[2] + o.mul(p.y, fb[3]), qpa);
  double bd, bp, bu, bv;
  if (!star) {
    const double m = o.mul(qd, qu), w = o.mul(m, bfen);
    const double G = bfm + bfmx * qu + bfmy * qv + bfen * E;
    bv = o.mul(m, bfmy + bfen * qv);
    const double y = o.div(w, by_d);
    bd = o.mul(qu, G) - y * e;
    bu = qd * G + m * bfmx + bfen * qp + w * qu;
    bp = bfmx + bfen * qu + o.div(y, qgm1);
    const double xu = o.div(bu, qna), xv = o.div(bv, qpa);
    const double x = xu * n.x + o.mul(xv, p.x), yy = xu * n.y + o.mul(xv, p.y);
    lb[0] = left ? bd : 0.0, lb[1] = left ? bp : 0.0, lb[2] = left ? x : 0.0, lb[3] = left ? yy : 0.0;
    rb[0] = left ? 0.0 : bd, rb[1] = left ? 0.0 : bp, rb[2] = left ? 0.0 : x, rb[3] = left ? 0.0 : yy;
    return;
  }
  double bss, bsk;
  {
    const auto qD = o.by(sk - ss), qJ = o.by(J);
    const double ds = o.div(J, qD), A = ss - qu, Q = o.div(qp, qJ), B = ss + Q;
    E += A * B;
    const double ps = qp + J * A, m = o.mul(ds, ss), w = o.mul(m, bfen);
    const double H = bfmx + bfen * ss, G = bfm + bfmx * ss + bfmy * qv + bfen * E;
    bv = o.mul(m, bfmy + bfen * qv);
    const double X = o.div(o.mul(ss, G), qD), wA = o.mul(w, A), Y = o.div(wA, qJ);
    const double S = X + H * A - Y * Q;
    const double y = o.div(w, by_d);
    bp = H + Y + o.div(y, qgm1);
    bd = o.mul(K, S) - y * e;
    const double qS = o.mul(qd, S), bA = o.mul(H, J) + w * B;
    bss = ds * G + m * bfmx + bfen * ps + bA + wA + ds * X;
    bu = w * qu - bA - qS;
    bsk = qS - ds * X;
  }
  // the wave speeds: ss = num/den, sl = min(lu - cL, ru - cR), sr = max(lu + cL, ru + cR)
  const double bnum = o.div(bss, qden);
  const double aL = o.mul(bnum, lu - ss), aR = o.mul(bnum, ru - ss);
  double bdL = tl * aL + (left ? bd : 0.0), bdR = (left ? 0.0 : bd) - tr * aR;
  double buL = dL * (bnum * tl - aL) + (left ? bu : 0.0), buR = (left ? 0.0 : bu) - dR * (bnum * tr - aR);
  double bpL = (left ? bp : 0.0) - bnum, bpR = (left ? 0.0 : bp) + bnum;
  const double bsl = aL * dL + (left ? bsk : 0.0), bsr = (left ? 0.0 : bsk) - aR * dR;
  double bcL, bcR;
  if (!sl_right && sr_right) {
    buL += bsl;
    buR += bsr;
    bcL = -bsl;
    bcR = bsr;
  } else if (sl_right && sr_right) {  // both waves from the right side, or the left, or crossed
    buR = add_here(add_here(buR, bsl), bsr);
    bcL = 0.0;
    bcR = add_here(bsr, -bsl);
  } else if (!sl_right) {
    buL = add_here(add_here(buL, bsl), bsr);
    bcL = add_here(bsr, -bsl);
    bcR = 0.0;
  } else {
    buR = add_here(buR, bsl);
    buL = add_here(buL, bsr);
    bcL = bsr;
    bcR = -bsl;
  }
  // c = sqrt(gamma p/d)
  const double hL = o.half(o.div(bcL, qdL)), hR = o.half(o.div(bcR, qdR));
  bdL -= hL * cL;
  bdR -= hR * cR;
  bpL += o.div(o.mul(hL, g), o.by(cL));
  bpR += o.div(o.mul(hR, g), o.by(cR));
  // rotation into the face frame: u = v.n/|n|, v_t = v.par/|par|
  const double xL = o.div(buL, qna), xR = o.div(buR, qna), xv = o.div(bv, qpa);
  const double vx = o.mul(xv, p.x), vy = o.mul(xv, p.y);
  lb[0] = bdL;
  lb[1] = bpL;
  lb[2] = xL * n.x + (left ? vx : 0.0);
  lb[3] = xL * n.y + (left ? vy : 0.0);
  rb[0] = bdR;
  rb[1] = bpR;
  rb[2] = xR * n.x + (left ? 0.0 : vx);
  rb[3] = xR * n.y + (left ? 0.0 : vy);
}
#else
// Reverse of primitive conversion, rotation into the face frame, Hllc
// (hllc.cpp:97-154, massflux, face at rest) and the rotation back: from fb
// (adjoint of {mass, energy, px, py}) to the adjoints of the two states.
// A call of its own: inlined, the compiler contracts other pairs of these
// products, and the FP32 gradients differ in the last bits from what they were
// (16.4 us a call, 14.9 inlined, at 256^2; 15.9 in blocks of 128).
__device__ __noinline__ void hllc_reverse(real g, rv2 n, real na, rv2 p, real pa, const real L[4], const real R[4],
                                          const real fb[4], real lb[4], real rb[4]) {
  // forward values
  const real dL = L[0], pL = L[1], dR = R[0], pR = R[1];
  const real eL = quot(quot(pL, dL), g - real(1)), cL = root(quot(g * pL, dL));
  const real eR = quot(quot(pR, dR), g - real(1)), cR = root(quot(g * pR, dR));
  const real lu = quot(L[2] * n.x + L[3] * n.y, na), lv = quot(L[2] * p.x + L[3] * p.y, pa);
  const real ru = quot(R[2] * n.x + R[3] * n.y, na), rv = quot(R[2] * p.x + R[3] * p.y, pa);
  const bool sl_right = (ru - cR) < (lu - cL);
  const real sl = sl_right ? ru - cR : lu - cL;
  const bool sr_right = (lu + cL) < (ru + cR);
  const real sr = sr_right ? ru + cR : lu + cL;
  const real num = pR - pL + dL * lu * (sl - lu) - dR * ru * (sr - ru);
  const real den = dL * (sl - lu) - dR * (sr - ru);
  const real ss = quot(num, den);
  const bool left = sl > 0 || (sl <= 0 && ss >= 0);
  const bool star = left ? !(sl > 0) : !(sr < 0);
  const real qd = left ? dL : dR, qp = left ? pL : pR, qe = left ? eL : eR;
  const real qu = left ? lu : ru, qv = left ? lv : rv, sk = left ? sl : sr;
  const real k2 = qu * qu + qv * qv;
  const real ek = qd * (real(0.5) * k2 + qe);
  // adjoint of the face-frame flux {fm, fmx, fmy, fen}
  const real bfm = fb[0], bfen = fb[1];
  const real bfmx = quot(n.x * fb[2] + n.y * fb[3], na);
  const real bfmy = quot(p.x * fb[2] + p.y * fb[3], pa);
  real bd = 0, bp = 0, bu = 0, bv = 0, be = 0, bek = 0, bsk = 0, bss = 0;
  if (star) {
    // ds = qd K/D, use = ek ds/qd + ds A B with K = sk - qu, D = sk - ss,
    // A = ss - qu, B = ss + Q, Q = qp/(qd K); fluxes gain sk*(u* - u)
    const real K = sk - qu, D = sk - ss;
    const real ds = quot(qd * K, D);
    const real Q = quot(quot(qp, qd), K);
    const real A = ss - qu, B = ss + Q;
    const real use = quot(ek * ds, qd) + ds * A * B;
    bsk += bfm * (ds - qd) + bfmx * (ds * ss - qu * qd) + bfmy * (ds * qv - qv * qd) + bfen * (use - ek);
    real bds = (bfm + bfmx * ss + bfmy * qv) * sk;
    bd -= (bfm + bfmx * qu + bfmy * qv) * sk;
    bu -= bfmx * qd * sk;
    bv += bfmy * (ds - qd) * sk;
    bss += bfmx * ds * sk;
    const real buse = bfen * sk;
    bek -= bfen * sk;
    bek += quot(buse * ds, qd);
    bds += buse * (quot(ek, qd) + A * B);
    bd -= quot(buse * ek * ds, qd * qd);
    const real bA = buse * ds * B, bB = buse * ds * A;
    bss += bA + bB;
    bu -= bA;
    bp += quot(bB, qd * K);
    bd -= quot(bB * Q, qd);
    real bK = quot(-bB * Q, K);
    bd += quot(bds * K, D);
    bK += quot(bds * qd, D);
    const real bD = quot(-bds * ds, D);
    bsk += bK + bD;
    bu -= bK;
    bss -= bD;
  }
  // physical flux along the normal: fm = qd qu, fmx = qp + qu qd qu,
  // fmy = qv qd qu, fen = (ek + qp) qu; ek = qd (|v|^2/2 + qe)
  bd += bfm * qu + bfmx * qu * qu + bfmy * qv * qu;
  bu += bfm * qd + real(2.0) * bfmx * qd * qu + bfmy * qv * qd + bfen * (ek + qp);
  bv += bfmy * qd * qu;
  bp += bfmx + bfen * qu;
  bek += bfen * qu;
  bd += bek * (real(0.5) * k2 + qe);
  bu += bek * qd * qu;
  bv += bek * qd * qv;
  be += bek * qd;
  // distribute to the chosen side, then the wave-speed paths
  real bdL = 0, bpL = 0, buL = 0, bvL = 0, beL = 0, bcL = 0;
  real bdR = 0, bpR = 0, buR = 0, bvR = 0, beR = 0, bcR = 0;
  real bsl = 0, bsr = 0;
  if (left) {
    bdL = bd, bpL = bp, buL = bu, bvL = bv, beL = be, bsl = bsk;
  } else {
    bdR = bd, bpR = bp, buR = bu, bvR = bv, beR = be, bsr = bsk;
  }
  // ss = num/den
  const real bnum = quot(bss, den), bden = quot(-bss * ss, den);
  bpR += bnum;
  bpL -= bnum;
  bdL += bnum * lu * (sl - lu) + bden * (sl - lu);
  buL += bnum * dL * (sl - real(2.0) * lu) - bden * dL;
  bsl += (bnum * lu + bden) * dL;
  bdR -= bnum * ru * (sr - ru) + bden * (sr - ru);
  buR -= bnum * dR * (sr - real(2.0) * ru) - bden * dR;
  bsr -= (bnum * ru + bden) * dR;
  // sl = min(lu - cL, ru - cR), sr = max(lu + cL, ru + cR)
  if (sl_right) {
    buR += bsl;
    bcR -= bsl;
  } else {
    buL += bsl;
    bcL -= bsl;
  }
  if (sr_right) {
    buR += bsr;
    bcR += bsr;
  } else {
    buL += bsr;
    bcL += bsr;
  }
  // e = p/(d (gamma-1)), c = sqrt(gamma p/d)
  bpL += quot(beL, dL * (g - real(1))) + quot(bcL * g, real(2.0) * cL * dL);
  bdL -= quot(beL * eL, dL) + quot(bcL * cL, real(2.0) * dL);
  bpR += quot(beR, dR * (g - real(1))) + quot(bcR * g, real(2.0) * cR * dR);
  bdR -= quot(beR * eR, dR) + quot(bcR * cR, real(2.0) * dR);
  // rotation into the face frame: u = v.n/|n|, v_t = v.par/|par|
  lb[0] = bdL;
  lb[1] = bpL;
  lb[2] = quot(buL * n.x, na) + quot(bvL * p.x, pa);
  lb[3] = quot(buL * n.y, na) + quot(bvL * p.y, pa);
  rb[0] = bdR;
  rb[1] = bpR;
  rb[2] = quot(buR * n.x, na) + quot(bvR * p.x, pa);
  rb[3] = quot(buR * n.y, na) + quot(bvR * p.y, pa);
}

#endif  // RG_ADJ_FP64

__device__ __forceinline__ void face_state(const AdjArgs& a, int pid, rv2 dm, real c[4]) {
  const int sid = source_of(a.mesh, pid);
  real gx[4], gy[4];
  load_r(a.cells, sid, c);
  load_r(a.slopes, 2 * sid, gx);
  load_r(a.slopes, 2 * sid + 1, gy);
#pragma unroll
  for (int q = 0; q < 4; ++q) c[q] = c[q] + gx[q] * dm.x + gy[q] * dm.y;
}

// One face; false (nothing stored) where its operands are outside O's range.
template <class O>
__device__ __forceinline__ bool face_reverse(O& o, const AdjArgs& a, const double* ubar, int e) {
  const MeshDev& m = a.mesh;
  const int2 fc = m.face_cells[e];
  // the transposed gather of the extensive update stays in FP64
  const double s = a.dt * a.geom.area[e];
  double fbd[4] = {0, 0, 0, 0};
  if (fc.y < m.n) load_raw(ubar, fc.y, fbd);
  if (fc.x < m.n) {
    double u[4];
    load_raw(ubar, fc.x, u);
#pragma unroll
    for (int q = 0; q < 4; ++q) fbd[q] -= u[q];
  }
  real fb[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) fb[q] = to_real(scaled(o, fbd[q], s));
  real L[4], R[4], lb[4], rb[4];
  face_state(a, fc.x, side_dm(a, e, true), L);
  face_state(a, fc.y, side_dm(a, e, false), R);
#if RG_ADJ_FP64
  hllc_reverse(o, a.gamma, a.gm1, r2(a.geom.nrm[e]), a.geom.nabs[e], r2(a.geom.par[e]), a.geom.area[e], L, R, fb, lb,
               rb);
  if (!o.ok) return false;
#else
  hllc_reverse(to_real(a.gamma), r2(a.g32.nrm[e]), a.g32.nabs[e], r2(a.g32.par[e]), a.g32.area[e], L, R, fb, lb, rb);
#endif
  store_r(a.side_bar, 2 * e, lb);
  store_r(a.side_bar, 2 * e + 1, rb);
  return true;
}

#if RG_ADJ_FP64
static __device__ __noinline__ void face_reverse_plain(const AdjArgs& a, const double* ubar, int e) {
  PlainOps o;
  face_reverse(o, a, ubar, e);
}
// One thread per face.  Bound by the FP64 unit (80 operations a warp) with the
// products and quotients on the integer pipes beside it.  Six blocks of 128 per
// SM (80 registers, 400 bytes spilt) hold most of a 256^2 mesh's faces at once:
// 48 us, against 51 with five, 50 with four and 52-58 in blocks of 256 and 512.
// 256^2 (132,000 faces) 123 -> 48 us.
__global__ void __launch_bounds__(kFaceBlock, 6) k_adj_faces(AdjArgs a, const double* ubar) {
  chain_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.mesh.e) return;
  RevOps o;
  if (!face_reverse(o, a, ubar, e)) face_reverse_plain(a, ubar, e);
}
#else
__global__ void __launch_bounds__(kFaceBlock) k_adj_faces(AdjArgs a, const double* ubar) {
  chain_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.mesh.e) return;
  int none = 0;
  face_reverse(none, a, ubar, e);
}
#endif

// a b + c d, the product that is rounded by itself fixed
__device__ __forceinline__ real dot2(real a, real b, real c, real d) {
#if RG_ADJ_FP64
  return fma(a, b, c * d);
#else
  return fmaf(a, b, __fmul_rn(c, d));
#endif
}
// Four lanes per cell, one component each: nothing passes between them, a
// quad's loads and stores are its cell's records, and a 256^2 mesh gives every
// SM 54 warps where a thread per cell gave 13 and waited for memory.  An entry
// that also takes the limiter's share is stored again after the loop: an add
// under the loop's test would cost the FP64 unit its clocks on every entry.
// 256^2: FP64 48 -> 34 us (its unit 80 % busy before), FP32 20 -> 8.3 us.
__global__ void __launch_bounds__(kBlock) k_adj_cell(AdjArgs a) {
  chain_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t >> 2, q = t & 3;
  const MeshDev& m = a.mesh;
  if (i >= m.n) return;
  const Trace& tr = static_cast<const Trace*>(a.trace)[i];
  const int b = m.cell_off[i], nn = m.cell_off[i + 1] - b;
  const int code = tr.code[q];
  // face-state adjoints -> state adjoint w and slope adjoints bx, by
  real w = 0, bx = 0, by = 0;
  for (int k = a.side_off[i], end = a.side_off[i + 1]; k < end; ++k) {
    const int s = a.sides[k];
    const rv2 dm = side_dm(a, s >> 1, !(s & 1));
    const real sb = static_cast<const real*>(a.side_bar)[4 * static_cast<size_t>(s) + q];
    w += sb;
    bx += sb * dm.x;
    by += sb * dm.y;
  }
  // limiter: s = naive*psi
  real bnx = bx, bny = by, extra = 0;
  int ex_at = -1;
  if ((code & 0xff) != kTraceNone) {
    const int k = code & 0xff, kind = (code >> 8) & 3;
    const real psi = tr.psi[q];
    bnx = bx * psi;
    bny = by * psi;
    if (kind != 3) {  // else clamped to zero: no dependence
      // psi = N/D with D = naive_x dm.x + naive_y dm.y (the centroid difference)
      // and N = coef*(W[neighbour] - W[cell])
      const real nx = tr.naive[q], ny = tr.naive[4 + q];
      const real bpsi = dot2(bx, nx, by, ny);
      const real D = tr.dphi[q];
      const real bN = quot(bpsi, D), bD = quot(-bpsi * psi, D);
      const rv2 dm = entry_dm(a, b + k);
      bnx = dot2(bD, dm.x, bx, psi);
      bny = dot2(bD, dm.y, by, psi);
      ex_at = (code >> 16) - 1;
      if (ex_at >= 0) {
        const real coef = kind == 2 ? to_real(a.theta) : real(1);
        extra = coef * bN;
        w -= extra;
      }
    }
  }
  // naive slope: nx = vx*mi.x + vy*mi.y, ny = vx*mi.z + vy*mi.w,
  // v = sum_k h_k (W[cell] + W[neighbour k])
  real mi[4];
  load_minv(a, i, mi);
  const real bvx = dot2(bnx, mi[0], bny, mi[2]), bvy = dot2(bnx, mi[1], bny, mi[3]);
  real* out = static_cast<real*>(a.entry_bar) + 4 * static_cast<size_t>(b) + q;
  real at = 0;
  for (int k = 0; k < nn; ++k) {
    const rv2 h = entry_h(a, b + k);
    const real c = dot2(bvx, h.x, bvy, h.y);
    w += c;
    if (ex_at == k) at = c;
    out[4 * k] = c;
  }
  if (ex_at >= 0) out[4 * ex_at] = at + extra;
  static_cast<real*>(a.self_bar)[t] = w;
}

// (all in FP64; the shares and the state are records of the working precision)
__global__ void __launch_bounds__(kBlock) k_adj_update(AdjArgs a, const double* ubar_in, double* ubar_out,
                                                       double* grad) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (i >= m.n) return;
  double w[4];
  load_wide(a.self_bar, i, w);
  for (int k = a.target_off[i]; k < a.target_off[i + 1]; ++k) {
    double c[4];
    load_wide(a.entry_bar, a.targets[k], c);
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] += c[q];
  }
  double ub[4];
  load_raw(ubar_in, i, ub);
  const double V = m.cd_volume[i];
  if (grad) {
    // U_0 = I(W_0): mass = V d, E = V p/(gamma-1) + V d |v|^2/2, P = mass v
    double c[4];
    load_wide(a.cells, i, c);
    const double k2 = c[2] * c[2] + c[3] * c[3];
    const double mass = V * c[0];
    double g[4];
    g[0] = w[0] + V * (ub[0] + 0.5 * k2 * ub[1] + c[2] * ub[2] + c[3] * ub[3]);
    g[1] = w[1] + quot(V, a.gamma - 1) * ub[1];
    g[2] = w[2] + mass * (c[2] * ub[1] + ub[2]);
    g[3] = w[3] + mass * (c[3] * ub[1] + ub[3]);
    store_raw(grad, i, g);
    return;
  }
  double u[4];
  load_raw(a.ext, i, u);
  cell_update_transpose(a.gamma, V, u, w, ub);
  store_raw(ubar_out, i, ub);
}

inline long long blocks(long long n) { return (n + kBlock - 1) / kBlock; }

}  // namespace

#if RG_ADJ_FP64
cudaError_t adj_launch_check(const AdjArgs& a, cudaStream_t s) {
  const int n = a.mesh.m > a.mesh.n ? a.mesh.m : a.mesh.n;
  k_adj_check<<<static_cast<unsigned>(blocks(n)), kBlock, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t adj_launch_seed(const AdjArgs& a, const double* wbar, double* ubar, cudaStream_t s) {
  chain(s, blocks(a.mesh.n), kBlock, k_adj_seed, a, wbar, ubar);
  return cudaGetLastError();
}

cudaError_t adj_launch_reverse(const AdjArgs& a, const double* ubar_in, double* ubar_out, double* grad,
                               cudaStream_t s) {
  chain(s, (a.mesh.e + kFaceBlock - 1) / kFaceBlock, kFaceBlock, k_adj_faces, a, ubar_in);
  chain(s, blocks(4 * static_cast<long long>(a.mesh.n)), kBlock, k_adj_cell, a);
  chain(s, blocks(a.mesh.n), kBlock, k_adj_update, a, ubar_in, ubar_out, grad);
  return cudaGetLastError();
}
#else
cudaError_t adj_launch_reverse32(const AdjArgs& a, const double* ubar_in, double* ubar_out, double* grad,
                                 cudaStream_t s) {
  chain(s, (a.mesh.e + kFaceBlock - 1) / kFaceBlock, kFaceBlock, k_adj_faces, a, ubar_in);
  chain(s, blocks(4 * static_cast<long long>(a.mesh.n)), kBlock, k_adj_cell, a);
  chain(s, blocks(a.mesh.n), kBlock, k_adj_update, a, ubar_in, ubar_out, grad);
  return cudaGetLastError();
}
#endif

}  // namespace rg
